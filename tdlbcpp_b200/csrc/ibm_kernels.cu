// Immersed-boundary forcing (Rushton-turbine markers) for sm_100a.
//
// Reference semantics (tdlbcpp/src/Forcing.hpp:56-176): markers are applied
// one after another in list order. Each marker
//   1. weights its 3x3 stencil in the i-k plane with the 3-point smoothed
//      delta (calcWeight, :18-35), indices wrapping periodically in i and k;
//   2. interpolates rho and (j + F/2) with the CURRENT F, i.e. including the
//      updates of earlier markers that share a cell (:91-121);
//   3. subtracts rho_sum * (uDelta, vDelta, wDelta) (:126-128);
//   4. spreads F = alpha*F - beta*w*sum into its 9 cells (:131-155).
// Cells no marker touched end with F = 0 (:162-174).
//
// Parallel form with the same result: a marker only interacts with markers
// of the same j-plane that share a stencil cell. The scheduler (schedule.cu, for
// the blades tdlb_runtime.hpp) assigns each marker a level = 1 + the highest level of an earlier marker sharing a
// cell, so markers of one level touch disjoint cells and every pair that
// shares a cell keeps its list order. One CTA per j-plane walks its levels
// with a barrier between them.
//
// "F = 0 where untouched" needs no full-grid sweep: the touched cells of each
// pass are recorded as one bit per cell (mask_new). The step kernel reads F
// only where the bit is set, and the next pass treats F as zero where neither
// the previous pass (mask_old) nor the current one has touched the cell.
//
// Per pass (launch_ibm): k_ibm_gather (everything the pass reads from the
// state: moments and starting F of every unique stencil cell of the static
// markers, weights and stencil moments of the blade markers; it also starts
// mask_new as the static touched flags), then k_ibm_spread (one plane per
// block: the static markers' levels on an F tile in shared memory, then the
// plane's blade levels on a shared-memory hash table of its blade cells). Planes
// with many cells (an impeller disk) take a 512-thread launch on the side
// stream; a tank that has those, or more blade markers in a plane than an
// ordinary block has threads, walks the blades with k_ibm_blades afterwards.
// The batched passes run the same steps per lattice.
#include "tdlb_kernels.cuh"
#include "tdlb_rotate.hpp"

#include <algorithm>
#include <map>
#include <mutex>
#include <utility>

namespace tdlb {

// 3-point smoothed delta (Forcing.hpp:18-35). The reference evaluates it
// in double (its literals promote the float argument) and rounds the result
// to float; every operation here is an explicitly rounded double operation
// in the reference's order, so no kernel can contract it differently and
// the weights equal the reference's bit for bit.
__device__ __forceinline__ float calc_weight(float xf) {
    const double x = (double)fabsf(xf);
    if (x > 1.5) return 0.f;
    double w;
    if (x <= 0.5) {
        const double r = __dsqrt_rn(__dadd_rn(__dmul_rn(__dmul_rn(-3.0, x), x), 1.0));
        w = __dmul_rn(1.0 / 3.0, __dadd_rn(1.0, r));
    } else {
        const double y = __dsub_rn(1.0, x);
        const double r = __dsqrt_rn(__dadd_rn(__dmul_rn(-3.0, __dmul_rn(y, y)), 1.0));
        w = __dmul_rn(1.0 / 6.0, __dsub_rn(__dsub_rn(5.0, __dmul_rn(3.0, x)), r));
    }
    return __double2float_rn(w);
}

// Weight of stencil offset (i1, k1) for a marker at fractions (icf, kcf):
// the product of the two 1-D weights, rounded to float (Forcing.hpp:37-48).
__device__ __forceinline__ float stencil_weight(float icf, float kcf, int i1, int k1) {
    return __fmul_rn(calc_weight(__fadd_rn(-icf, (float)i1)), calc_weight(__fadd_rn(-kcf, (float)k1)));
}

__device__ __forceinline__ int wrap_i(int a, int n) { return a < 0 ? a + n : (a >= n ? a - n : a); }

template <typename S>
__device__ __forceinline__ float ld_state(const float* plane, long long e) {
    if constexpr (sizeof(S) == 4) return plane[e];
    else return Storage<S>::dec(reinterpret_cast<const S*>(plane)[e]);
}

// rho and momentum of the state at interior cell (i, j, k). With a residual
// box, a cell near it adds the residuals of its locations inside the box
// after its 18 loads (the other cells take no box code).
template <typename S>
__device__ __forceinline__ void cell_moments4(const Planes& A, int mode, int even, const Dims& g, int i, int j, int k,
                                              const CollideParams& p, float* m4, const ResidualBox& rb) {
    if (mode == 1) {
        const long long e = g.at(i, j, k);
#pragma unroll
        for (int s = 0; s < 4; s++) m4[s] = ld_state<S>(A.p[s], e);
        return;
    }
    float q[NQ];
    const bool near_box = Storage<S>::deviation && rb.near(i, j, k);
    if (mode == 0) {
#pragma unroll
        for (int d = 0; d < NQ; d++) {
            const int si = i - cx_of(d), sj = j - cy_of(d), sk = k - cz_of(d);
            const bool in = (unsigned)si < (unsigned)g.nx && (unsigned)sj < (unsigned)g.ny && (unsigned)sk < (unsigned)g.nz;
            const long long src = in ? g.at(si, sj, sk) : g.at(i, j, k);
            q[d] = ld_state<S>(A.p[d], src) + (Storage<S>::deviation ? (is_face(d) ? p.wface : p.wedge) : 0.f);
        }
        if (near_box) {   // residual box: the exact deviations
#pragma unroll
            for (int d = 0; d < NQ; d++) {
                const int si = i - cx_of(d), sj = j - cy_of(d), sk = k - cz_of(d);
                const bool in = (unsigned)si < (unsigned)g.nx && (unsigned)sj < (unsigned)g.ny && (unsigned)sk < (unsigned)g.nz;
                const int li = in ? si : i, lj = in ? sj : j, lk = in ? sk : k;
                if (rb.contains(li, lj, lk)) q[d] += *rb.at(d, li, lj, lk);
            }
        }
        moments4_of(q, m4);
        return;
    }
    const int i1 = i + 1 == g.nx ? 0 : i + 1, j1 = j + 1 == g.ny ? 0 : j + 1, k1 = k + 1 == g.nz ? 0 : k + 1;
    const int nread = mode == 3 ? 4 : NQ;
#pragma unroll
    for (int d = 0; d < NQ; d++) {
        if (d >= nread) break;
        const int s = even ? d : (d ^ 1);
        const int sg = even ? -1 : 1;
        const bool oi = sg * cx_of(s) > 0, oj = sg * cy_of(s) > 0, ok = sg * cz_of(s) > 0;
        q[d] = ld_state<S>(A.p[s], g.at(oi ? i1 : i, oj ? j1 : j, ok ? k1 : k)) +
               (mode == 2 && Storage<S>::deviation ? (is_face(d) ? p.wface : p.wedge) : 0.f);
    }
    if (mode == 2 && near_box) {   // residual box: the exact deviations
#pragma unroll
        for (int d = 0; d < NQ; d++) {
            const int s = even ? d : (d ^ 1);
            const int sg = even ? -1 : 1;
            const bool oi = sg * cx_of(s) > 0, oj = sg * cy_of(s) > 0, ok = sg * cz_of(s) > 0;
            if (rb.contains(oi ? i1 : i, oj ? j1 : j, ok ? k1 : k)) q[d] += *rb.at(s, oi ? i1 : i, oj ? j1 : j, ok ? k1 : k);
        }
    }
    if (mode == 3) {
#pragma unroll
        for (int s = 0; s < 4; s++) m4[s] = q[s];
    } else {
        moments4_of(q, m4);
    }
}

// ---------------------------------------------------------------------------
// First segment (markers that do not move), prepared once per upload.
// ---------------------------------------------------------------------------
__global__ void k_ibm_prepare(IbmArgs a, float* __restrict__ prep) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n0) return;
    const Marker mk = a.markers[a.sched[p]];
    float* row = prep + (size_t)p * PF_STRIDE;
    int c = 0;
    for (int k1 = -1; k1 <= 1; k1++)
        for (int i1 = -1; i1 <= 1; i1++, c++)
            row[PF_W + c] = stencil_weight(mk.iCartFraction, mk.kCartFraction, i1, k1);
    row[PF_U] = mk.uDelta;
    row[PF_V] = mk.vDelta;
    row[PF_WV] = mk.wDelta;
}

// Per pass: rho and momentum of every unique stencil cell of the first
// segment, and the F each cell starts the pass with (zero unless the previous
// pass touched it, Forcing.hpp:162-174).
template <typename S>
__device__ __forceinline__ void ibm_cell(const IbmArgs& a, int e, float4& m, float4& f) {
    const Dims& g = a.g;
    const int row = e / g.jp;
    const int j = e - row * g.jp;
    const int i = row / g.nz;
    const int k = row - i * g.nz;
    float m4[4];
    cell_moments4<S>(a.A, a.state_mode, a.even, g, i, j, k, a.p, m4, a.rbox);
    m = make_float4(m4[0], m4[1], m4[2], m4[3]);
    const bool live = (a.mask_old[(long long)row * g.jw + (j >> 5)] >> (j & 31)) & 1u;
    f = live ? a.F4[e] : make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ void put_cell(const IbmArgs& a, int c, const float4 m, const float4 f) {
    const long long C = a.ncell;
    reinterpret_cast<float4*>(a.cell_m)[c] = m;
    a.cell_F[c] = f.x;
    a.cell_F[C + c] = f.y;
    a.cell_F[2 * C + c] = f.z;
}

// The cells of 32 consecutive planes, 8 list places of each: place p of plane
// j is cell plane_cell[j] + p, the places sorted by (i, k). The markers of a
// tank repeat from plane to plane, so place p is the same (i, k) in
// neighbouring planes and lanes that run over the planes read whole lines of
// every population row; a tile in shared memory then turns the results round
// so that lanes running over the places write the lists (128 bytes of a list
// per plane). Any list is right; one that does not repeat reads a sector per
// cell and row. Bound by DRAM bytes: 72 populations + 16 F + 4 index + 28
// written per cell (400^3: 64 us for 2.1 M cells). Planes with more than
// skip_above cells (an impeller disk, whose cells fill an (i, k) area of a single
// j) are taken in list order instead.
constexpr int kGatherThreads = 32 * kCellPlaces;
struct CellTile {
    int e[32][kCellPlaces + 1];
    float4 m[kCellPlaces][33];
    float4 f[kCellPlaces][33];
};
template <typename S>
__device__ __forceinline__ void ibm_cell_tile(const IbmArgs& a, CellTile& sm, int j0, int p0, int skip_above) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    {
        const int jj = threadIdx.x / kCellPlaces, p = threadIdx.x % kCellPlaces;
        int e = -1;
        if (j0 + jj < a.g.ny) {
            const int c0 = a.plane_cell[j0 + jj], nc = a.plane_cell[j0 + jj + 1] - c0;
            if (nc <= skip_above && p0 + p < nc) e = a.cell_e[c0 + p0 + p];
        }
        sm.e[jj][p] = e;
    }
    __syncthreads();
    const int e = sm.e[lane][warp];
    if (e >= 0) {
        float4 m, f;
        ibm_cell<S>(a, e, m, f);
        sm.m[warp][lane] = m;
        sm.f[warp][lane] = f;
    }
    __syncthreads();
    const int jj = threadIdx.x / kCellPlaces, p = threadIdx.x % kCellPlaces;
    if (sm.e[jj][p] >= 0) put_cell(a, a.plane_cell[j0 + jj] + p0 + p, sm.m[p][jj], sm.f[p][jj]);
}
// Second segment (the blades): weight and moments of stencil cell c of blade
// marker t, u = c * ntail + t (c = 3 (k1 + 1) + (i1 + 1)): the nine cells of a
// marker are gathered in parallel; c = 0 also writes the marker velocity.
template <typename S>
__device__ __forceinline__ void ibm_tail_cell(const IbmArgs& a, int u) {
    const int ntail = a.n - a.n0;
    if (u >= 9 * ntail) return;
    const int c = u / ntail, t = u - c * ntail;
    const Marker mk = a.markers[a.sched[a.n0 + t]];
    const int k1 = c / 3 - 1, i1 = c - 3 * (c / 3) - 1;
    const int i2 = wrap_i((int)mk.i + i1, a.g.nx), j = (int)mk.j, k2 = wrap_i((int)mk.k + k1, a.g.nz);
    float m4[4];
    cell_moments4<S>(a.A, a.state_mode, a.even, a.g, i2, j, k2, a.p, m4, a.rbox);
    float* s = a.tail;
    const long long cap = a.tail_cap;
    s[(TF_W + c) * cap + t] = stencil_weight(mk.iCartFraction, mk.kCartFraction, i1, k1);
    s[(TF_RHO + c) * cap + t] = m4[0];
    s[(TF_MX + c) * cap + t] = m4[1];
    s[(TF_MY + c) * cap + t] = m4[2];
    s[(TF_MZ + c) * cap + t] = m4[3];
    s[(TF_CELL + c) * cap + t] = __int_as_float((i2 << 16) | k2);
    if (c == 0) {
        s[TF_U * cap + t] = mk.uDelta;
        s[TF_V * cap + t] = mk.vDelta;
        s[TF_WV * cap + t] = mk.wDelta;
    }
}

// Everything the pass reads from the state, in one launch: the blades' stencils
// (the first tail_blocks blocks), the big planes' cells (big_blocks blocks of each),
// the other planes' cell tiles; its threads also start mask_new as the first
// segment's touched flags (mask_static, a multiple of 16 bytes).
template <typename S>
__global__ void __launch_bounds__(kGatherThreads) k_ibm_gather(IbmArgs a, int tail_blocks, int big_blocks, int tiles_j) {
    __shared__ CellTile sm;
    after_previous();
    {
        const int n4 = (int)(a.mask_bytes / 16);
        for (int w = (int)(blockIdx.x * blockDim.x + threadIdx.x); w < n4; w += (int)(gridDim.x * blockDim.x))
            reinterpret_cast<uint4*>(a.mask_new)[w] = reinterpret_cast<const uint4*>(a.mask_static)[w];
    }
    int b = (int)blockIdx.x;
    if (b < tail_blocks) return ibm_tail_cell<S>(a, b * kGatherThreads + (int)threadIdx.x);
    b -= tail_blocks;
    if (b < a.n_big * big_blocks) {
        const int j = a.plane_list[a.n_small + b / big_blocks];
        const int c = a.plane_cell[j] + b % big_blocks * kGatherThreads + (int)threadIdx.x;
        if (c >= a.plane_cell[j + 1]) return;
        float4 m, f;
        ibm_cell<S>(a, a.cell_e[c], m, f);
        return put_cell(a, c, m, f);
    }
    b -= a.n_big * big_blocks;
    ibm_cell_tile<S>(a, sm, b % tiles_j * 32, b / tiles_j * kCellPlaces, a.smem_cells);
}

// Bulk asynchronous copies global -> shared memory with an mbarrier
// (cp.async.bulk, no multicast): one thread issues them, the group waits on
// the barrier's transaction count. Source and destination 16-byte aligned,
// sizes a multiple of 16 bytes.
__device__ unsigned g_ibm_bulk_timeouts = 0;   // waits that gave up (then the tile is loaded by plain loads)

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t* bar, unsigned bytes) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(smem_addr(bar)),
                 "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_to_smem(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(smem_addr(bar)) : "memory");
}
// Wait for phase 0 of the barrier, at most `limit` polls; false when it gave up.
__device__ __forceinline__ bool mbar_wait0(uint64_t* bar, int limit) {
    for (int it = 0; it < limit; it++) {
        unsigned done;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0; selp.u32 %0, 1, 0, p; }"
                     : "=r"(done) : "r"(smem_addr(bar)) : "memory");
        if (done) return true;
    }
    return false;
}
// The 16-byte aligned span of elements [c0, c0 + n) of a 4-byte array:
// the first element copied, its offset from c0 and the bytes to copy.
struct BulkSpan {
    const void* src;
    int off;
    unsigned bytes;
};
__device__ __forceinline__ BulkSpan bulk_span(const void* base, int c0, int n) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(base) + 4ull * (unsigned)c0;
    const uintptr_t lo = a & ~uintptr_t(15), hi = (a + 4ull * (unsigned)n + 15) & ~uintptr_t(15);
    return BulkSpan{reinterpret_cast<const void*>(lo), (int)((a - lo) >> 2), (unsigned)(hi - lo)};
}
// Floats between the three F arrays of a bulk tile of `cells` cells: room
// for the 16-byte rounding of each copy, and a multiple of 4, so that every
// array (a bulk copy's destination) starts on a 16-byte boundary.
__host__ __device__ constexpr int bulk_tile_stride(int cells) { return (cells + 8 + 3) & ~3; }

// Element i of a row held as float4 registers (i a compile-time constant
// after unrolling).
template <int N>
__device__ __forceinline__ float f4_lane(const float4 (&r)[N], int i) {
    const float4 v = r[i >> 2];
    return (i & 3) == 0 ? v.x : (i & 3) == 1 ? v.y : (i & 3) == 2 ? v.z : v.w;
}

// Bring elements [c0, c0 + n) of a 4-byte array into L2 (cp.async.bulk
// prefetch: no completion to wait for). The span is rounded out to 16 bytes;
// every array prefetched this way is allocated with 16 elements of padding.
__device__ __forceinline__ void prefetch_l2(const void* base, int c0, int n) {
    if (n <= 0) return;
    const BulkSpan sp = bulk_span(base, c0, n);
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(sp.src), "r"(sp.bytes) : "memory");
}
// The per-marker and per-cell data the walk of plane j reads, into L2 while the
// block fills its tile: the first segment's rows (slots [p0, p1)), the plane's
// cell moments and elements, and the blade markers' gathered stencils (slots
// [q0, q1) of the second segment). One array per lane.
__device__ __forceinline__ void prefetch_plane(const IbmArgs& a, int c0, int nc, int p0, int p1, int q0, int q1) {
    const int lane = threadIdx.x;
    if (lane >= 32) return;
    for (int f = lane; f < 3 + TF_COUNT; f += 32) {
        if (f == 0) prefetch_l2(a.prep, p0 * PF_STRIDE, (p1 - p0) * PF_STRIDE);
        else if (f == 1) prefetch_l2(a.cell_m, 4 * c0, 4 * nc);
        else if (f == 2) prefetch_l2(a.cell_e, c0, nc);
        else prefetch_l2(a.tail + (size_t)(f - 3) * a.tail_cap, q0 - a.n0, q1 - q0);
    }
}

// Slot offsets of a plane's levels [lv0, lv1]: the first kLevelSmem staged in
// shared memory, so that a level starts without a trip to the L2.
constexpr int kLevelSmem = 64;
struct Levels {
    const int* global;   // a.level_ptr + lv0
    const int* staged;
    int n;               // levels
    __device__ __forceinline__ int at(int l) const { return l < kLevelSmem ? staged[l] : __ldg(global + l); }
};
template <int NT>
__device__ __forceinline__ Levels stage_levels(const IbmArgs& a, const int* plane_lv, int j, int* staged) {
    const int lv0 = plane_lv[j], n = plane_lv[j + 1] - lv0;
    for (int l = threadIdx.x; l < kLevelSmem && l <= n; l += NT) staged[l] = a.level_ptr[lv0 + l];
    return Levels{a.level_ptr + lv0, staged, n};
}

// Blade levels of plane j on global memory: F and the touched flags are
// read back from L2 (__ldcg), since earlier levels of this CTA wrote them.
// Used when the plane's blade stencils do not fit the shared-memory table;
// a called function rather than inlined, so that this rare fallback costs
// the register-bound walks around it no registers.
template <int NT>
__device__ __noinline__ void blade_levels_global(const IbmArgs& a, int j) {
    const Dims g = a.g;
    const float* s = a.tail;
    const long long cap = a.tail_cap;
    for (int lv = a.plane_lv1[j]; lv < a.plane_lv1[j + 1]; lv++) {
        const int p0 = a.level_ptr[lv], p1 = a.level_ptr[lv + 1];
#pragma unroll 1
        for (int p = p0 + (int)threadIdx.x; p < p1; p += NT) {
            const int t = p - a.n0;
            float rhoSum = 0.f, xSum = 0.f, ySum = 0.f, zSum = 0.f;
#pragma unroll
            for (int c = 0; c < 9; c++) {
                const float w = s[(TF_W + c) * cap + t];
                const int packed = __float_as_int(s[(TF_CELL + c) * cap + t]);
                const int i2 = packed >> 16, k2 = packed & 0xffff;
                const long long e = g.at(i2, j, k2), wd = g.word(i2, j, k2);
                const uint32_t bit = 1u << (j & 31);
                const bool live = (__ldcg(a.mask_new + wd) & bit) || (a.mask_old[wd] & bit);
                const float4 v = live ? __ldcg(a.F4 + e) : make_float4(0.f, 0.f, 0.f, 0.f);
                const float vx = v.x, vy = v.y, vz = v.z;
                rhoSum = fmaf(w, s[(TF_RHO + c) * cap + t], rhoSum);
                xSum = fmaf(w, fmaf(0.5f, vx, s[(TF_MX + c) * cap + t]), xSum);
                ySum = fmaf(w, fmaf(0.5f, vy, s[(TF_MY + c) * cap + t]), ySum);
                zSum = fmaf(w, fmaf(0.5f, vz, s[(TF_MZ + c) * cap + t]), zSum);
            }
            xSum = fmaf(-rhoSum, s[TF_U * cap + t], xSum);
            ySum = fmaf(-rhoSum, s[TF_V * cap + t], ySum);
            zSum = fmaf(-rhoSum, s[TF_WV * cap + t], zSum);
            a.sums[p] = xSum;
            a.sums[a.n + p] = ySum;
            a.sums[2 * a.n + p] = zSum;
#pragma unroll
            for (int c = 0; c < 9; c++) {
                const int packed = __float_as_int(s[(TF_CELL + c) * cap + t]);
                const int i2 = packed >> 16, k2 = packed & 0xffff;
                const long long e = g.at(i2, j, k2), wd = g.word(i2, j, k2);
                const uint32_t bit = 1u << (j & 31);
                const bool live = (__ldcg(a.mask_new + wd) & bit) || (a.mask_old[wd] & bit);
                const float4 v = live ? __ldcg(a.F4 + e) : make_float4(0.f, 0.f, 0.f, 0.f);
                const float bw = a.beta * s[(TF_W + c) * cap + t];
                a.F4[e] = make_float4(fmaf(a.alpha, v.x, -bw * xSum), fmaf(a.alpha, v.y, -bw * ySum),
                                      fmaf(a.alpha, v.z, -bw * zSum), 0.f);
                atomicOr(&a.mask_new[wd], bit);
            }
        }
        __syncthreads();
    }
}

// The table of blade_levels_tile and the update of one marker on it.
struct BladeTable {
    int* keys;
    float *hx, *hy, *hz;
};
struct BladeMarker {
    float w[9], rho[9], mx[9], my[9], mz[9], u, v, wv;
    __device__ __forceinline__ void load(const float* s, long long cap, int t) {
#pragma unroll
        for (int c = 0; c < 9; c++) {
            w[c] = s[(TF_W + c) * cap + t];
            rho[c] = s[(TF_RHO + c) * cap + t];
            mx[c] = s[(TF_MX + c) * cap + t];
            my[c] = s[(TF_MY + c) * cap + t];
            mz[c] = s[(TF_MZ + c) * cap + t];
        }
        u = s[TF_U * cap + t];
        v = s[TF_V * cap + t];
        wv = s[TF_WV * cap + t];
    }
    // interpolate at the table entries hh, subtract the marker's velocity,
    // spread; the sums go to slot p
    __device__ __forceinline__ void apply(const IbmArgs& a, const BladeTable& h, const int (&hh)[9], int p, bool distinct) const {
        float rhoSum = 0.f, xSum = 0.f, ySum = 0.f, zSum = 0.f;
        float ox[9], oy[9], oz[9];
#pragma unroll
        for (int c = 0; c < 9; c++) {
            ox[c] = h.hx[hh[c]];
            oy[c] = h.hy[hh[c]];
            oz[c] = h.hz[hh[c]];
            rhoSum = fmaf(w[c], rho[c], rhoSum);
            xSum = fmaf(w[c], fmaf(0.5f, ox[c], mx[c]), xSum);
            ySum = fmaf(w[c], fmaf(0.5f, oy[c], my[c]), ySum);
            zSum = fmaf(w[c], fmaf(0.5f, oz[c], mz[c]), zSum);
        }
        xSum = fmaf(-rhoSum, u, xSum);
        ySum = fmaf(-rhoSum, v, ySum);
        zSum = fmaf(-rhoSum, wv, zSum);
        a.sums[p] = xSum;
        a.sums[a.n + p] = ySum;
        a.sums[2 * a.n + p] = zSum;
        if (distinct) {   // 9 different cells: independent updates
#pragma unroll
            for (int c = 0; c < 9; c++) {
                const float bw = a.beta * w[c];
                h.hx[hh[c]] = fmaf(a.alpha, ox[c], -bw * xSum);
                h.hy[hh[c]] = fmaf(a.alpha, oy[c], -bw * ySum);
                h.hz[hh[c]] = fmaf(a.alpha, oz[c], -bw * zSum);
            }
        } else {
#pragma unroll
            for (int c = 0; c < 9; c++) {   // sequential: a wrapped stencil sees its own update
                const float bw = a.beta * w[c];
                h.hx[hh[c]] = fmaf(a.alpha, h.hx[hh[c]], -bw * xSum);
                h.hy[hh[c]] = fmaf(a.alpha, h.hy[hh[c]], -bw * ySum);
                h.hz[hh[c]] = fmaf(a.alpha, h.hz[hh[c]], -bw * zSum);
            }
        }
    }
};

// Blade levels of plane j on a shared-memory table. The plane's 9 x nb
// stencil references (nb blade markers) go into an open-addressing hash
// table keyed by the packed cell (i << 16 | k), H >= 9 nb entries of (key,
// Fx, Fy, Fz), so every insert ends within H probes. Each cell's F is loaded
// once -- zero unless this pass (mask_new: the first segment's cells) or the
// previous one touched it -- the levels run on the table, and the cells go
// back to F with their touched flags. The walk reads and writes the same
// values in the same order as blade_levels_global; only the L2 round trips
// between levels go. Needs blade_table_words(nb) words of `tile`; returns
// false, having done nothing, when they do not fit.
// With a thread for every marker (nb <= NT) a thread holds its marker's data
// and table entries in registers from the start, and the thread that put a
// cell into the table loads its F and writes it back, so a level is table
// reads, the update and a barrier, and the walk one trip to the L2 before
// them. (Bound by latency. 160^3 tank, 84 markers a plane: 17 us with the data
// of each level loaded inside it.)
template <int NT>
__device__ __forceinline__ bool blade_levels_tile(const IbmArgs& a, int j, float* tile, int tile_words, const Levels lv) {
    const int q0 = lv.at(0), nb = lv.at(lv.n) - q0, nref = 9 * nb;
    int lg = 5;
    while ((1 << lg) < nref) lg++;
    const int H = 1 << lg;
    if (4LL * H + nref > (long long)tile_words) return false;
    BladeTable h{reinterpret_cast<int*>(tile), tile + H, tile + 2 * H, tile + 3 * H};
    const Dims g = a.g;
    const float* s = a.tail;
    const long long cap = a.tail_cap;
    const bool distinct = g.nx >= 3 && g.nz >= 3;   // the 9 stencil cells of a marker differ
    const int tid = (int)threadIdx.x;
    // the entry of `key`; first: this call put it there
    auto insert = [&](int key, bool& first) {
        unsigned at = ((unsigned)key * 2654435761u) >> (32 - lg);
        first = false;
        for (int probe = 0; probe < H; probe++) {
            const int prev = atomicCAS(&h.keys[at], -1, key);
            first = prev == -1;
            if (first || prev == key) break;
            at = (at + 1) & (unsigned)(H - 1);
        }
        return (int)at;
    };
    // F of `key`, zero unless this pass or the previous one touched it
    auto load_cell = [&](int key, float& x, float& y, float& z) {
        const int i2 = key >> 16, k2 = key & 0xffff;
        const long long wd = g.word(i2, j, k2);
        const uint32_t bit = 1u << (j & 31);
        const float4 v = __ldcg(a.F4 + g.at(i2, j, k2));   // (a lattice cell whatever the flags say)
        const bool live = ((__ldcg(a.mask_new + wd) | a.mask_old[wd]) & bit) != 0u;
        x = live ? v.x : 0.f;
        y = live ? v.y : 0.f;
        z = live ? v.z : 0.f;
    };
    auto store_cell = [&](int key, int at) {
        const int i2 = key >> 16, k2 = key & 0xffff;
        a.F4[g.at(i2, j, k2)] = make_float4(h.hx[at], h.hy[at], h.hz[at], 0.f);
        atomicOr(&a.mask_new[g.word(i2, j, k2)], 1u << (j & 31));
    };

    if (nb <= NT) {
        const bool on = tid < nb;
        const int t = q0 + tid - a.n0;
        BladeMarker mk;
        int key[9], hh[9];
        if (on) {
#pragma unroll
            for (int c = 0; c < 9; c++) key[c] = __float_as_int(s[(TF_CELL + c) * cap + t]);
            mk.load(s, cap, t);
        }
        for (int e = tid; e < H; e += NT) h.keys[e] = -1;
        __syncthreads();
        unsigned mine = 0;
        if (on) {
            // every cell's F, so that the loads leave together; the inserts
            // meanwhile say which of them this thread keeps
            float x[9], y[9], z[9];
#pragma unroll
            for (int c = 0; c < 9; c++) load_cell(key[c], x[c], y[c], z[c]);
#pragma unroll
            for (int c = 0; c < 9; c++) {
                bool first;
                hh[c] = insert(key[c], first);
                mine |= first ? 1u << c : 0u;
            }
#pragma unroll
            for (int c = 0; c < 9; c++)
                if ((mine >> c) & 1u) {
                    h.hx[hh[c]] = x[c];
                    h.hy[hh[c]] = y[c];
                    h.hz[hh[c]] = z[c];
                }
        }
        __syncthreads();
        for (int l = 0; l < lv.n; l++) {
            const int p = q0 + tid;
            if (p >= lv.at(l) && p < lv.at(l + 1)) mk.apply(a, h, hh, p, distinct);
            __syncthreads();
        }
        if (on) {
#pragma unroll
            for (int c = 0; c < 9; c++)
                if ((mine >> c) & 1u) store_cell(key[c], hh[c]);
        }
        return true;
    }
    int* ref = reinterpret_cast<int*>(tile + 4 * H);
    for (int e = tid; e < H; e += NT) h.keys[e] = -1;
    __syncthreads();
    for (int r = tid; r < nref; r += NT) {
        const int m = r / 9, c = r - 9 * m;
        bool first;
        ref[r] = insert(__float_as_int(s[(TF_CELL + c) * cap + (q0 + m - a.n0)]), first);
    }
    __syncthreads();
    for (int e = tid; e < H; e += NT)
        if (h.keys[e] >= 0) load_cell(h.keys[e], h.hx[e], h.hy[e], h.hz[e]);
    __syncthreads();
    for (int l = 0; l < lv.n; l++) {
        const int p1 = lv.at(l + 1);
#pragma unroll 1
        for (int p = lv.at(l) + tid; p < p1; p += NT) {
            BladeMarker mk;
            mk.load(s, cap, p - a.n0);
            int hh[9];
#pragma unroll
            for (int c = 0; c < 9; c++) hh[c] = ref[9 * (p - q0) + c];
            mk.apply(a, h, hh, p, distinct);
        }
        __syncthreads();
    }
    for (int e = tid; e < H; e += NT)
        if (h.keys[e] >= 0) store_cell(h.keys[e], e);
    return true;
}

// A first-segment marker's data: its slot row (weights, places, velocity) and,
// gathered through the row's places, its cells' rho and momentum.
struct SlotRow {
    float4 r[PF_STRIDE / 4];
    __device__ __forceinline__ void load(const float* prep, int p) {
#pragma unroll
        for (int u = 0; u < PF_STRIDE / 4; u++) r[u] = __ldg(reinterpret_cast<const float4*>(prep + (size_t)p * PF_STRIDE) + u);
    }
    __device__ __forceinline__ float w(int c) const { return f4_lane(r, PF_W + c); }
    __device__ __forceinline__ int place(int c) const { return __float_as_int(f4_lane(r, PF_CELL + c)); }
};
struct SlotMoments {
    float4 m[9];
    __device__ __forceinline__ void load(const float4* cm, const SlotRow& row) {
#pragma unroll
        for (int c = 0; c < 9; c++) m[c] = cm[row.place(c)];
    }
};
__device__ __forceinline__ void apply_slot(const IbmArgs& a, const SlotRow& row, const SlotMoments& mo, float* fx, float* fy,
                                           float* fz, int p, bool distinct) {
    float rhoSum = 0.f, xSum = 0.f, ySum = 0.f, zSum = 0.f;
    float ox[9], oy[9], oz[9];
#pragma unroll
    for (int c = 0; c < 9; c++) {
        const int li = row.place(c);
        const float w = row.w(c);
        ox[c] = fx[li];
        oy[c] = fy[li];
        oz[c] = fz[li];
        rhoSum = fmaf(w, mo.m[c].x, rhoSum);
        xSum = fmaf(w, fmaf(0.5f, ox[c], mo.m[c].y), xSum);
        ySum = fmaf(w, fmaf(0.5f, oy[c], mo.m[c].z), ySum);
        zSum = fmaf(w, fmaf(0.5f, oz[c], mo.m[c].w), zSum);
    }
    xSum = fmaf(-rhoSum, f4_lane(row.r, PF_U), xSum);
    ySum = fmaf(-rhoSum, f4_lane(row.r, PF_V), ySum);
    zSum = fmaf(-rhoSum, f4_lane(row.r, PF_WV), zSum);
    a.sums[p] = xSum;
    a.sums[a.n + p] = ySum;
    a.sums[2 * a.n + p] = zSum;
    if (distinct) {
        // 9 different cells: each update starts from the value read above, so
        // the 27 stores are independent
#pragma unroll
        for (int c = 0; c < 9; c++) {
            const int li = row.place(c);
            const float bw = a.beta * row.w(c);
            fx[li] = fmaf(a.alpha, ox[c], -bw * xSum);
            fy[li] = fmaf(a.alpha, oy[c], -bw * ySum);
            fz[li] = fmaf(a.alpha, oz[c], -bw * zSum);
        }
    } else {
#pragma unroll
        for (int c = 0; c < 9; c++) {   // sequential: a wrapped stencil sees its own update
            const int li = row.place(c);
            const float bw = a.beta * row.w(c);
            fx[li] = fmaf(a.alpha, fx[li], -bw * xSum);
            fy[li] = fmaf(a.alpha, fy[li], -bw * ySum);
            fz[li] = fmaf(a.alpha, fz[li], -bw * zSum);
        }
    }
}

// One block per j-plane: the plane's first-segment levels on an F tile in
// shared memory (planes with more cells than the tile holds work on cell_F in
// place), write-back to F, then (BLADES) the blade levels, on a shared-memory
// table when they fit the tile, else on global F. The touched flags of the
// first segment never change, so each pass starts mask_new as a copy of them
// (mask_static) and the blade walk adds its cells. The tile is
// [3][bulk_tile_stride(tile_cells)] words (F x, y, z), filled by bulk copies of
// the plane's cell range.
//
// A level is a chain -- its markers read the F that the levels before it wrote --
// so the walk is bound by latency, and everything but F is brought in ahead:
// the level offsets are staged, a thread's next slot row is on its way two
// slots ahead and the next slot's cell moments one slot ahead (PIPE: 84 more
// registers, launches of 128 threads; the 512 threads of a big plane hold only
// their current slot and hide the trips by number). Measured on B200 with the
// rows one slot ahead and the moments loaded inside the level: 37 us for a
// 160^3 tank, 85 us at 400^3.
template <int NT, bool PIPE, bool BLADES>
__device__ __forceinline__ void ibm_spread_plane(const IbmArgs& a, int j, int tile_cells, float* tile) {
    __shared__ uint64_t bar;
    __shared__ int fail;
    __shared__ int staged0[kLevelSmem], staged1[BLADES ? kLevelSmem : 1];
    const int tid = (int)threadIdx.x;
    const int c0 = a.plane_cell[j], nc = a.plane_cell[j + 1] - c0;
    const Levels lv = stage_levels<NT>(a, a.plane_lv0, j, staged0);
    Levels lb{nullptr, nullptr, 0};
    if (BLADES) lb = stage_levels<NT>(a, a.plane_lv1, j, staged1);
    const long long C = a.ncell;
    const bool in_smem = nc <= tile_cells;
    float *fx, *fy, *fz;
    int at_x = 0, at_y = 0, at_z = 0;   // the arrays' first words in the tile
    if (in_smem && nc > 0) {
        const int tc = bulk_tile_stride(tile_cells);
        const BulkSpan sx = bulk_span(a.cell_F + c0, 0, nc), sy = bulk_span(a.cell_F + C + c0, 0, nc),
                       sz = bulk_span(a.cell_F + 2 * C + c0, 0, nc);
        if (tid == 0) {
            mbar_init(&bar);
            fail = 0;
            mbar_expect(&bar, sx.bytes + sy.bytes + sz.bytes);
            bulk_to_smem(tile, sx.src, sx.bytes, &bar);
            bulk_to_smem(tile + tc, sy.src, sy.bytes, &bar);
            bulk_to_smem(tile + 2 * tc, sz.src, sz.bytes, &bar);
        }
        __syncthreads();   // the barrier is set up; the staged offsets are in
        prefetch_plane(a, c0, nc, lv.at(0), lv.at(lv.n), BLADES ? lb.at(0) : a.n0, BLADES ? lb.at(lb.n) : a.n0);
        at_x = sx.off;
        at_y = tc + sy.off;
        at_z = 2 * tc + sz.off;
        fx = tile + at_x; fy = tile + at_y; fz = tile + at_z;
    } else {
        __syncthreads();
        fx = a.cell_F + c0; fy = a.cell_F + C + c0; fz = a.cell_F + 2 * C + c0;
    }
    // ---- first segment: each marker in list order relative to every marker
    //      it shares a cell with (level walk). With x and z at least 3 the 9
    //      stencil cells of a marker differ (the stencil wraps onto itself
    //      only on a narrower lattice).
    const bool distinct = a.g.nx >= 3 && a.g.nz >= 3;
    const float4* cm = reinterpret_cast<const float4*>(a.cell_m) + c0;   // rho, jx, jy, jz
    // Rounds: the slots [b, b + NT) of a level, one per thread, round after
    // round, level after level (e: the level's end, where the next one starts).
    // Row and moment sets take turns (their roles, not their contents, move
    // on: a copied register would wait for its load).
    struct Round {
        int l, b, e;
    };
    auto after = [&](Round q) {
        q.b += NT;
        if (q.b >= q.e) {
            q.l++;
            q.b = q.e;
            if (q.l < lv.n) q.e = lv.at(q.l + 1);
        }
        return q;
    };
    Round q0{0, 0, 0}, q1 = q0, q2 = q0;   // (no slot: b + tid >= e)
    SlotRow r0, r1, r2;
    SlotMoments m0, m1;
    if (PIPE && lv.n > 0) {
        q0 = Round{0, lv.at(0), lv.at(1)};
        if (q0.b + tid < q0.e) r0.load(a.prep, q0.b + tid);
        q1 = after(q0);
        if (q1.b + tid < q1.e) r1.load(a.prep, q1.b + tid);
        q2 = after(q1);
        if (q0.b + tid < q0.e) m0.load(cm, r0);
    }
    if (in_smem && nc > 0) {
        // bounded wait; the block decides together whether it gave up, so
        // that every thread takes the same barriers
        if (!mbar_wait0(&bar, 1 << 20)) fail = 1;
        __syncthreads();
        if (fail) {
            // should not happen: count it, give the copies more time, then
            // load the tile with plain loads
            if (tid == 0) atomicAdd(&g_ibm_bulk_timeouts, 1u);
            mbar_wait0(&bar, 1 << 22);
            __syncthreads();
            for (int t = tid; t < nc; t += NT) {
                fx[t] = a.cell_F[c0 + t];
                fy[t] = a.cell_F[C + c0 + t];
                fz[t] = a.cell_F[2 * C + c0 + t];
            }
            __syncthreads();
        }
    }
    if (PIPE && in_smem) {
        float *sx = tile + at_x, *sy = tile + at_y, *sz = tile + at_z;   // shared memory, as the compiler can see
        // the round of (rc, mc); on the way: the next round's moments, the row after it
        auto round = [&](const SlotRow& rc, const SlotRow& rn, SlotRow& rnn, const SlotMoments& mc, SlotMoments& mn) {
            if (q1.b + tid < q1.e) mn.load(cm, rn);
            if (q2.b + tid < q2.e) rnn.load(a.prep, q2.b + tid);
            if (q0.b + tid < q0.e) apply_slot(a, rc, mc, sx, sy, sz, q0.b + tid, distinct);
            if (q1.l != q0.l) __syncthreads();
            q0 = q1;
            q1 = q2;
            q2 = after(q2);
            return q0.l < lv.n;
        };
        bool more = lv.n > 0;
        while (more) {
            if (!(more = round(r0, r1, r2, m0, m1))) break;
            if (!(more = round(r1, r2, r0, m1, m0))) break;
            if (!(more = round(r2, r0, r1, m0, m1))) break;
            if (!(more = round(r0, r1, r2, m1, m0))) break;
            if (!(more = round(r1, r2, r0, m0, m1))) break;
            more = round(r2, r0, r1, m1, m0);
        }
    } else {
        for (int l = 0; l < lv.n; l++) {
            const int p1 = lv.at(l + 1);
#pragma unroll 1
            for (int q = lv.at(l) + tid; q < p1; q += NT) {
                r0.load(a.prep, q);
                m0.load(cm, r0);
                apply_slot(a, r0, m0, fx, fy, fz, q, distinct);
            }
            __syncthreads();
        }
    }
    // ---- write the plane's cells back to F (eight element loads in flight
    //      per thread)
    {
        int t = tid;
        for (; t + 7 * NT < nc; t += 8 * NT) {
            int e[8];
#pragma unroll
            for (int u = 0; u < 8; u++) e[u] = a.cell_e[c0 + t + u * NT];
#pragma unroll
            for (int u = 0; u < 8; u++) a.F4[e[u]] = make_float4(fx[t + u * NT], fy[t + u * NT], fz[t + u * NT], 0.f);
        }
        for (; t < nc; t += NT) {
            const int e = a.cell_e[c0 + t];
            a.F4[e] = make_float4(fx[t], fy[t], fz[t], 0.f);
        }
    }
    // ---- second segment (blades), unless a separate launch walks them
    if constexpr (BLADES) {
        if (lb.n == 0) return;
        __syncthreads();
        if (!blade_levels_tile<NT>(a, j, tile, 3 * bulk_tile_stride(tile_cells), lb)) blade_levels_global<NT>(a, j);
    }
}

// A plane per block: the ordinary planes with 128 threads, the big ones (an
// impeller disk) with 512. Two blocks of 128 at most share an SM, which leaves
// registers and shared memory to the outer launch of a split step beside them
// (the walk's time is the chain's, not the number of threads').
template <int NT, bool BLADES>
__global__ void __launch_bounds__(NT, NT == 128 ? 2 : 1) k_ibm_spread(IbmArgs a, const int* __restrict__ planes,
                                                                     int tile_cells) {
    extern __shared__ __align__(128) float btile[];             // [3][bulk_tile_stride(tile_cells)]
    int b = (int)blockIdx.x;
    after_previous(b);
    ibm_spread_plane<NT, NT == 128, BLADES>(a, planes[b], tile_cells, btile);
}

// The blade levels of the planes that have blades, one plane per CTA of NT
// threads, after both first-segment spreads have written their planes' F, for
// planes with more blade markers than an ordinary plane's block has threads.
// `words` floats of shared memory hold the plane's hash table.
template <int NT>
__global__ void __launch_bounds__(NT, 1) k_ibm_blades(IbmArgs a, const int* __restrict__ planes, int nplanes,
                                                      int words) {
    extern __shared__ __align__(16) float btab[];
    __shared__ int staged[kLevelSmem];
    if ((int)blockIdx.x >= nplanes) return;
    const int j = planes[blockIdx.x];
    const Levels lv = stage_levels<NT>(a, a.plane_lv1, j, staged);
    __syncthreads();
    if (!blade_levels_tile<NT>(a, j, btab, words, lv)) blade_levels_global<NT>(a, j);
}

// Impeller rotation on the device: recomputes the blade markers of the
// resident list for a new angle (main.cpp:409-426 does this on the host and
// re-uploads the whole list every step).
__global__ void k_rotate_markers(const double* __restrict__ xz, Marker* __restrict__ out, int n, double ca, double sa,
                                 double omega, double ci, double ck, int nx, int nz) {
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    after_previous(q);
    if (q >= n) return;
    const RotatedMarker r = rotate_marker(xz[2 * q], xz[2 * q + 1], ca, sa, omega, ci, ck, nx, nz);
    Marker& m = out[q];
    m.i = r.i;
    m.k = r.k;
    m.iCartFraction = r.iCartFraction;
    m.kCartFraction = r.kCartFraction;
    m.uDelta = r.uDelta;
    m.vDelta = 0.f;
    m.wDelta = r.wDelta;
}

__global__ void __launch_bounds__(256) k_place_blades(const int* __restrict__ stage, int* __restrict__ markers, int mwords,
                                                      int* __restrict__ order, int n, int* __restrict__ level_ptr, int nlev,
                                                      int* __restrict__ plane_lv, int nplane) {
    int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    after_previous(t);
    const int total = mwords + n + nlev + nplane;
    if (t >= total) return;
    const int v = stage[t];
    if (t < mwords) markers[t] = v;
    else if ((t -= mwords) < n) order[t] = v;
    else if ((t -= n) < nlev) level_ptr[t] = v;
    else plane_lv[t - nlev] = v;
}

cudaError_t launch_place_blades(const int* stage, Marker* markers, int n, int* order, int* level_ptr, int nlev, int* plane_lv,
                                int nplane, cudaStream_t st) {
    const int mwords = (int)(sizeof(Marker) / sizeof(int)) * n;
    return launch_chained(k_place_blades, (mwords + n + nlev + nplane + 255) / 256, 256, 0, st, stage,
                          reinterpret_cast<int*>(markers), mwords, order, n, level_ptr, nlev, plane_lv, nplane);
}

cudaError_t launch_rotate_markers(const double* xz, Marker* out, int n, double ca, double sa, double omega, double ci,
                                  double ck, int nx, int nz, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    return launch_chained(k_rotate_markers, (n + 255) / 256, 256, 0, st, xz, out, n, ca, sa, omega, ci, ck, nx, nz);
}

// FP64 sums of five values over a block of 256 threads (fixed order: a warp's
// lanes by halves, then the warps by halves), in thread 0.
__device__ __forceinline__ void block_sum5(double (&v)[5]) {
    __shared__ double part[8][5];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int w = 16; w > 0; w /= 2)
#pragma unroll
        for (int c = 0; c < 5; c++) v[c] += __shfl_down_sync(0xffffffffu, v[c], w);
    if (lane == 0)
#pragma unroll
        for (int c = 0; c < 5; c++) part[warp][c] = v[c];
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int c = 0; c < 5; c++) v[c] = lane < 8 ? part[lane][c] : 0.0;
#pragma unroll
        for (int w = 4; w > 0; w /= 2)
#pragma unroll
            for (int c = 0; c < 5; c++) v[c] += __shfl_down_sync(0xffffffffu, v[c], w);
    }
    __syncthreads();
}

// Deterministic FP64 reduction of the marker forces over the impeller's slots
// (a list built with the schedule: 4 % of a 400^3 tank's markers): fixed grid,
// fixed strides and trees; the block that finishes last adds the blocks' sums
// the same way. One launch bound by latency; with a pass over every marker, a
// second launch and one thread adding 128 blocks' sums it was 26 us at 400^3, 13 us
// at 24^3. counter: zero before, and again after.
__global__ void __launch_bounds__(256) k_marker_load(IbmArgs a, const int* __restrict__ slots, int n, double ci, double ck,
                                                     double* partial, unsigned* counter, double* out) {
    __shared__ bool last;
    int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    after_previous(t);
    double acc[5] = {0, 0, 0, 0, 0};
    for (; t < n; t += gridDim.x * blockDim.x) {
        const int p = slots[t];
        const Marker mk = a.markers[a.sched[p]];
        const double fx = -(double)a.beta * (double)a.sums[p];
        const double fy = -(double)a.beta * (double)a.sums[a.n + p];
        const double fz = -(double)a.beta * (double)a.sums[2 * a.n + p];
        const double di = (double)mk.i + (double)mk.iCartFraction - ci;
        const double dk = (double)mk.k + (double)mk.kCartFraction - ck;
        acc[0] += fx;
        acc[1] += fy;
        acc[2] += fz;
        acc[3] += dk * fx - di * fz;   // (r x F) along j, r = (di, 0, dk)
        acc[4] += 1.0;
    }
    block_sum5(acc);
    if (gridDim.x > 1) {
        if (threadIdx.x == 0) {
#pragma unroll
            for (int c = 0; c < 5; c++) partial[blockIdx.x * 5 + c] = acc[c];
            __threadfence();
            last = atomicAdd(counter, 1u) == gridDim.x - 1;
        }
        __syncthreads();
        if (!last) return;
        __threadfence();
#pragma unroll
        for (int c = 0; c < 5; c++) acc[c] = threadIdx.x < gridDim.x ? __ldcg(partial + threadIdx.x * 5 + c) : 0.0;
        block_sum5(acc);
        if (threadIdx.x == 0) *counter = 0u;
    }
    if (threadIdx.x == 0)
        for (int c = 0; c < 5; c++) out[c] = acc[c];
}

// The slots whose marker is the impeller's (list index >= begin), in slot
// order: two passes over 256-slot groups, counts then places.
__global__ void __launch_bounds__(256) k_impeller_slots(const int* __restrict__ sched, int n, int begin, int* __restrict__ offset,
                                                        int* __restrict__ slots) {
    __shared__ int warps[8];
    const int p = (int)(blockIdx.x * 256 + threadIdx.x), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool in = p < n && sched[p] >= begin;
    const unsigned vote = __ballot_sync(0xffffffffu, in);
    if (lane == 0) warps[warp] = __popc(vote);
    __syncthreads();
    int before = 0, all = 0;
    for (int w = 0; w < 8; w++) {
        if (w < warp) before += warps[w];
        all += warps[w];
    }
    if (!slots) {
        if (threadIdx.x == 0) offset[blockIdx.x] = all;
    } else if (in) {
        slots[offset[blockIdx.x] + before + __popc(vote & ((1u << lane) - 1u))] = p;
    }
}

cudaError_t launch_impeller_slots(const int* sched, int n, int begin, int* offset, int* slots, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_impeller_slots<<<(n + 255) / 256, 256, 0, st>>>(sched, n, begin, offset, slots);
    return cudaGetLastError();
}

// Ordered sum of the block partials: the warp stages them in shared memory
// (coalesced, all loads in flight at once), then one thread adds them in
// block order, so the result does not depend on the launch.
template <int NC, int NB>
__device__ __forceinline__ void ordered_final(const double* __restrict__ partial, int nblocks, double* out) {
    __shared__ double v[NB * NC];
    const int n = nblocks * NC;
    for (int q = threadIdx.x; q < n; q += blockDim.x) v[q] = partial[q];
    __syncthreads();
    if (threadIdx.x != 0) return;
    double acc[NC];
#pragma unroll
    for (int c = 0; c < NC; c++) acc[c] = 0.0;
    for (int b = 0; b < nblocks; b++)
#pragma unroll
        for (int c = 0; c < NC; c++) acc[c] += v[b * NC + c];
#pragma unroll
    for (int c = 0; c < NC; c++) out[c] = acc[c];
}

cudaError_t launch_marker_load(const IbmArgs& a, const int* slots, int n, double ci, double ck, double* partial,
                               unsigned* counter, double* out, cudaStream_t st) {
    const int blocks = n <= 0 ? 1 : std::min(kLoadBlocks, (n + 511) / 512);   // two slots a thread, more in a large tank
    return launch_chained(k_marker_load, blocks, 256, 0, st, a, slots, n, ci, ck, partial, counter, out);
}

// FP64 mass and momentum over all interior cells, deterministic: a fixed
// grid of kReduceBlocks blocks, a fixed per-thread stride, a fixed tree,
// then one thread sums the block partials in order.
template <typename S>
__global__ void __launch_bounds__(256) k_reduce_fp64(IbmArgs a, const uint32_t* __restrict__ mask, double* partial) {
    __shared__ double red[4][256];
    const Dims g = a.g;
    const long long total = g.cells();
    double acc[4] = {0, 0, 0, 0};
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        g.cell(t, i, j, k);
        float m4[4];
        cell_moments4<S>(a.A, a.state_mode, a.even, g, i, j, k, a.p, m4, a.rbox);
        const long long e = g.at(i, j, k);
        const bool on = (mask[g.word(i, j, k)] >> (j & 31)) & 1u;
        acc[0] += m4[0];
        const float4 f = on ? a.F4[e] : make_float4(0.f, 0.f, 0.f, 0.f);
        acc[1] += (double)m4[1] + (on ? 0.5 * (double)f.x : 0.0);
        acc[2] += (double)m4[2] + (on ? 0.5 * (double)f.y : 0.0);
        acc[3] += (double)m4[3] + (on ? 0.5 * (double)f.z : 0.0);
    }
    for (int c = 0; c < 4; c++) red[c][threadIdx.x] = acc[c];
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w)
            for (int c = 0; c < 4; c++) red[c][threadIdx.x] += red[c][threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int c = 0; c < 4; c++) partial[blockIdx.x * 4 + c] = red[c][0];
}

__global__ void k_reduce_fp64_final(const double* partial, int nblocks, double* out) {
    ordered_final<4, kReduceBlocks>(partial, nblocks, out);
}

cudaError_t launch_reduce_fp64(const IbmArgs& a, const uint32_t* mask, double* partial, double* out, cudaStream_t st) {
    with_storage(a.storage, [&](auto s) {
        k_reduce_fp64<decltype(s)><<<kReduceBlocks, 256, 0, st>>>(a, mask, partial);
    });
    k_reduce_fp64_final<<<1, 32, 0, st>>>(partial, kReduceBlocks, out);
    return cudaGetLastError();
}

// Rest state of the 16-bit storage at density rho: every population
// w_d * rho, stored as its deviation from w_d * rho0.
template <typename S>
__global__ void k_fill_rest(Planes Q, long long plane, float rho_ratio_m1, CollideParams p) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= plane) return;
#pragma unroll
    for (int d = 0; d < NQ; d++)
        reinterpret_cast<S*>(Q.p[d])[t] = Storage<S>::enc(rho_ratio_m1 * (is_face(d) ? p.wface : p.wedge));
}

cudaError_t launch_fill_rest(Planes Q, long long plane, float rho, float rho0, int storage, const CollideParams& p,
                             cudaStream_t st) {
    const unsigned b = (unsigned)((plane + 255) / 256);
    const float r = rho / rho0 - 1.f;
    with_storage(storage, [&](auto s) { k_fill_rest<decltype(s)><<<b, 256, 0, st>>>(Q, plane, r, p); });
    return cudaGetLastError();
}

// The dynamic shared-memory limit is a per-kernel, per-device attribute that
// every lattice and batch shares: it only ever grows, so that a smaller
// lattice set up later cannot lower it below what a larger one launches with.
cudaError_t raise_smem_limit(const void* fn, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<const void*, int>, size_t> set;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    size_t& cur = set[{fn, dev}];
    if (bytes <= cur) return cudaSuccess;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) cur = bytes;
    return e;
}

// Shared memory (floats) of the blade launch for a plane of nb blade
// markers: blade_levels_tile's table of H >= 9 nb entries (a power of two,
// at least 32) of four words, and 9 nb references.
int blade_table_words(int nb) {
    const int nref = 9 * nb;
    int H = 32;
    while (H < nref) H *= 2;
    return 4 * H + nref;
}

cudaError_t ibm_prepare_blades(int words) {
    return raise_smem_limit((const void*)k_ibm_blades<512>, (size_t)words * sizeof(float));
}

// Shared memory of a plane's bulk tile of `big_cells` cells (none when the tile
// does not fit).
size_t big_bulk_bytes(int big_cells) { return big_cells > 0 ? (size_t)12 * bulk_tile_stride(big_cells) : 0; }

cudaError_t ibm_prepare_smem(int small_cells, size_t big_bytes) {
    const size_t small = big_bulk_bytes(small_cells);
    cudaError_t e = raise_smem_limit((const void*)k_ibm_spread<128, false>, small);
    if (e == cudaSuccess) e = raise_smem_limit((const void*)k_ibm_spread<128, true>, small);
    if (e == cudaSuccess) e = raise_smem_limit((const void*)k_ibm_spread<512, false>, big_bytes);
    return e;
}

cudaError_t launch_ibm_prepare(const IbmArgs& a, float* prep, cudaStream_t st) {
    if (a.n0 <= 0) return cudaSuccess;
    k_ibm_prepare<<<(a.n0 + 255) / 256, 256, 0, st>>>(a, prep);
    return cudaGetLastError();
}

cudaError_t launch_ibm(const IbmArgs& a, cudaStream_t st) {
    const int tail_blocks = (int)((9LL * (a.n - a.n0) + kGatherThreads - 1) / kGatherThreads);
    const int big_blocks = (a.max_big + kGatherThreads - 1) / kGatherThreads;
    const int tiles_j = (a.g.ny + 31) / 32;
    const long long blocks = tail_blocks + (long long)a.n_big * big_blocks +
                             (long long)tiles_j * ((a.max_cells + kCellPlaces - 1) / kCellPlaces);
    // (an empty list still starts mask_new)
    cudaError_t err = cudaSuccess;
    with_storage(a.storage, [&](auto s) {
        err = launch_chained(k_ibm_gather<decltype(s)>, (unsigned)std::max(blocks, 1LL), kGatherThreads, 0, st, a, tail_blocks,
                             big_blocks, tiles_j);
    });
    if (err != cudaSuccess) return err;
    // Side stream: the planes with many cells (an impeller disk), with a
    // full-size tile and 512 threads, beside the ordinary planes.
    if (a.n_big > 0) {
        err = cudaEventRecord(a.ev_fork, st);
        if (err == cudaSuccess) err = cudaStreamWaitEvent(a.side, a.ev_fork, 0);
        if (err != cudaSuccess) return err;
        k_ibm_spread<512, false><<<a.n_big, 512, big_bulk_bytes(a.big_tile_cells), a.side>>>(a, a.plane_list + a.n_small,
                                                                                        a.big_tile_cells);
        err = cudaGetLastError();
        if (err == cudaSuccess) err = cudaEventRecord(a.ev_join, a.side);
        if (err != cudaSuccess) return err;
    }
    // A plane's blades are walked by its own block when there is a thread for
    // every marker and no big plane has any; else by a launch of their own,
    // once every plane's first segment is in F.
    const bool own = a.blade_max <= 128 && a.n_big == 0;
    if (a.n_small > 0) {
        const size_t bytes = big_bulk_bytes(a.smem_cells);
        const auto kernel = own && a.n_blade > 0 ? k_ibm_spread<128, true> : k_ibm_spread<128, false>;
        err = launch_chained(kernel, a.n_small, 128, bytes, st, a, a.plane_list, a.smem_cells);
    }
    if (err == cudaSuccess && a.n_big > 0) err = cudaStreamWaitEvent(st, a.ev_join, 0);
    if (err != cudaSuccess || own || a.n_blade == 0) return err;
    k_ibm_blades<512><<<a.n_blade, 512, (size_t)a.blade_words * sizeof(float), st>>>(a, a.blade_planes, a.n_blade,
                                                                                  a.blade_words);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Batched passes: the immersed-boundary passes of many lattices in one set of
// launches. Every block takes one work item (lattice, first index); the
// lattice's IbmArgs is staged in shared memory and the single-lattice body
// runs on it, so each lattice's result equals its own launch_ibm.
// ---------------------------------------------------------------------------
template <int NT>
__device__ __forceinline__ void stage_args(IbmArgs& dst, const IbmArgs* src) {
    static_assert(sizeof(IbmArgs) % 8 == 0, "IbmArgs words");
    constexpr int words = sizeof(IbmArgs) / 8;
    for (int w = threadIdx.x; w < words; w += NT)
        reinterpret_cast<unsigned long long*>(&dst)[w] = reinterpret_cast<const unsigned long long*>(src)[w];
}

// What the pass reads from the states (k_ibm_gather), one work item per block.
template <typename S>
__global__ void __launch_bounds__(kGatherThreads) k_ibm_gather_batch(const IbmArgs* __restrict__ args,
                                                                     const int2* __restrict__ work) {
    __shared__ IbmArgs sa;
    __shared__ CellTile sm;
    const GatherItem w = GatherItem::of(work[blockIdx.x]);
    stage_args<kGatherThreads>(sa, args + w.tank);
    __syncthreads();
    if (w.kind == GATHER_TAIL) {
        ibm_tail_cell<S>(sa, w.y * kGatherThreads + (int)threadIdx.x);
    } else if (w.kind == GATHER_FLAGS) {
        const int n4 = (int)(sa.mask_bytes / 16), v0 = w.y * (kMaskCopyWords / 4);
        for (int v = v0 + (int)threadIdx.x; v < min(n4, v0 + kMaskCopyWords / 4); v += kGatherThreads)
            reinterpret_cast<uint4*>(sa.mask_new)[v] = reinterpret_cast<const uint4*>(sa.mask_static)[v];
    } else {
        ibm_cell_tile<S>(sa, sm, w.j0(), w.p0(), 0x7fffffff);
    }
}

// A work item (lattice, plane) per block, blades included: the ordinary planes
// with 128 threads, the big ones with 512.
template <int NT>
__global__ void __launch_bounds__(NT, NT == 128 ? 2 : 1) k_ibm_spread_batch(const IbmArgs* __restrict__ args,
                                                                           const int2* __restrict__ work) {
    extern __shared__ __align__(128) float btile[];
    __shared__ IbmArgs sa;
    const int2 w = work[blockIdx.x];
    stage_args<NT>(sa, args + w.x);
    __syncthreads();
    ibm_spread_plane<NT, NT == 128, true>(sa, w.y, NT == 128 ? sa.smem_cells : sa.big_tile_cells, btile);
}

cudaError_t ibm_batch_prepare_smem(int small_cells, int big_cells) {
    const cudaError_t e = raise_smem_limit((const void*)k_ibm_spread_batch<128>, big_bulk_bytes(small_cells));
    return e != cudaSuccess ? e : raise_smem_limit((const void*)k_ibm_spread_batch<512>, big_bulk_bytes(big_cells));
}

cudaError_t launch_ibm_batch(const IbmBatch& b, cudaStream_t st, cudaStream_t side, cudaEvent_t fork, cudaEvent_t join) {
    if (b.n_gather > 0) {
        with_storage(b.storage, [&](auto s) {
            k_ibm_gather_batch<decltype(s)><<<b.n_gather, kGatherThreads, 0, st>>>(b.args, b.gather);
        });
    }
    cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    if (b.n_big > 0) {
        err = cudaEventRecord(fork, st);
        if (err != cudaSuccess) return err;
        err = cudaStreamWaitEvent(side, fork, 0);
        if (err != cudaSuccess) return err;
        k_ibm_spread_batch<512><<<b.n_big, 512, big_bulk_bytes(b.big_tile), side>>>(b.args, b.big);
        err = cudaGetLastError();
        if (err != cudaSuccess) return err;
        err = cudaEventRecord(join, side);
        if (err != cudaSuccess) return err;
    }
    if (b.n_small > 0) k_ibm_spread_batch<128><<<b.n_small, 128, big_bulk_bytes(b.small_tile), st>>>(b.args, b.small);
    err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    if (b.n_big > 0) return cudaStreamWaitEvent(st, join, 0);
    return cudaSuccess;
}

}  // namespace tdlb
