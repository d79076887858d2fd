// Step-kernel templates (Simple pull and Esotwist in place), generic in the
// population storage type S (float, __half, __nv_bfloat16) and in V, the
// cells per thread. Instantiated by step_kernels.cu (FP32 storage) and
// step_kernels_h16.cu (16-bit deviation storage). See step_kernels.cu for
// the streaming semantics.
#pragma once
#include <cstring>

#include "tdlb_kernels.cuh"

namespace tdlb {

// ---------------------------------------------------------------------------
// Thread mapping shared by both schemes: V consecutive cells (along j) of one
// row per thread ("quad"), quads numbered row-major over (row, jq); a warp covers 32
// consecutive quads, so neighbouring lanes hold neighbouring cells of the
// same row except at row ends (where the wall rule or the periodic wrap
// applies anyway). V in {1, 2, 4}; populations move as float/float2/float4.
// ---------------------------------------------------------------------------
constexpr unsigned FULL = 0xffffffffu;

// FP32 vector helpers (F, Nu and FP32 populations)
template <int V>
__device__ __forceinline__ void vload(const float* __restrict__ p, float (&v)[V]) {
    if constexpr (V == 4) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(p));
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else if constexpr (V == 2) {
        const float2 t = __ldg(reinterpret_cast<const float2*>(p));
        v[0] = t.x; v[1] = t.y;
    } else {
        v[0] = __ldg(p);
    }
}
template <int V>
__device__ __forceinline__ void vstore(float* p, const float (&v)[V]) {
    if constexpr (V == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else if constexpr (V == 2) *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
    else *p = v[0];
}
// Streaming stores (st.global.cs: first out of L2), for data the kernel does
// not read again -- Simple's destination buffer and Nu, FP32 storage.
// Measured on B200 at 400^3: k_step_simple 1.554 -> 1.528-1.535 ms; the
// in-place Esotwist kernel, which stores to the lines it has just read,
// measured slower with them (1.676 -> 1.724 ms), and so did the 16-bit Simple
// step (1.541 -> 1.574 ms whole step); those keep plain stores.
template <int V>
__device__ __forceinline__ void vstore_cs(float* p, const float (&v)[V]) {
    if constexpr (V == 4) __stcs(reinterpret_cast<float4*>(p), make_float4(v[0], v[1], v[2], v[3]));
    else if constexpr (V == 2) __stcs(reinterpret_cast<float2*>(p), make_float2(v[0], v[1]));
    else __stcs(p, v[0]);
}

// Population plane access in storage type S: V elements from element e,
// decoded to FP32 (RO: read-only, non-coherent path).
template <typename S, int V, bool RO>
__device__ __forceinline__ void pload(const float* plane, int e, float (&v)[V]) {
    if constexpr (sizeof(S) == 4) {
        const float* p = plane + e;
        if constexpr (V == 4) {
            const float4 t = RO ? __ldg(reinterpret_cast<const float4*>(p)) : *reinterpret_cast<const float4*>(p);
            v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
        } else if constexpr (V == 2) {
            const float2 t = RO ? __ldg(reinterpret_cast<const float2*>(p)) : *reinterpret_cast<const float2*>(p);
            v[0] = t.x; v[1] = t.y;
        } else {
            v[0] = RO ? __ldg(p) : *p;
        }
    } else {
        const S* p = reinterpret_cast<const S*>(plane) + e;
        if constexpr (V == 4) {
            const uint2 t = RO ? __ldg(reinterpret_cast<const uint2*>(p)) : *reinterpret_cast<const uint2*>(p);
            S s4[4];
            memcpy(s4, &t, sizeof t);
#pragma unroll
            for (int k = 0; k < 4; k++) v[k] = Storage<S>::dec(s4[k]);
        } else if constexpr (V == 2) {
            const unsigned t = RO ? __ldg(reinterpret_cast<const unsigned*>(p)) : *reinterpret_cast<const unsigned*>(p);
            S s2[2];
            memcpy(s2, &t, sizeof t);
            v[0] = Storage<S>::dec(s2[0]);
            v[1] = Storage<S>::dec(s2[1]);
        } else {
            const unsigned short t = RO ? __ldg(reinterpret_cast<const unsigned short*>(p))
                                        : *reinterpret_cast<const unsigned short*>(p);
            S s1;
            memcpy(&s1, &t, sizeof t);
            v[0] = Storage<S>::dec(s1);
        }
    }
}
template <typename S, bool RO>
__device__ __forceinline__ float pload1(const float* plane, int e) {
    float v[1];
    pload<S, 1, RO>(plane, e, v);
    return v[0];
}
template <typename S, int V, bool CS = false>
__device__ __forceinline__ void pstore(float* plane, int e, const float (&v)[V]) {
    if constexpr (sizeof(S) == 4) {
        if constexpr (CS) vstore_cs<V>(plane + e, v);
        else vstore<V>(plane + e, v);
    } else {
        S* p = reinterpret_cast<S*>(plane) + e;
        if constexpr (V == 4) {
            S s4[4];
#pragma unroll
            for (int k = 0; k < 4; k++) s4[k] = Storage<S>::enc(v[k]);
            uint2 t;
            memcpy(&t, s4, sizeof t);
            if constexpr (CS) __stcs(reinterpret_cast<uint2*>(p), t);
            else *reinterpret_cast<uint2*>(p) = t;
        } else if constexpr (V == 2) {
            S s2[2] = {Storage<S>::enc(v[0]), Storage<S>::enc(v[1])};
            unsigned t;
            memcpy(&t, s2, sizeof t);
            if constexpr (CS) __stcs(reinterpret_cast<unsigned*>(p), t);
            else *reinterpret_cast<unsigned*>(p) = t;
        } else {
            if constexpr (CS) {
                const S enc = Storage<S>::enc(v[0]);
                unsigned short t;
                memcpy(&t, &enc, sizeof t);
                __stcs(reinterpret_cast<unsigned short*>(p), t);
            } else {
                *p = Storage<S>::enc(v[0]);
            }
        }
    }
}
template <typename S>
__device__ __forceinline__ void pstore1(float* plane, int e, float v) {
    const float a[1] = {v};
    pstore<S, 1>(plane, e, a);
}
// rest-population offset of direction/slot d in the deviation storage
template <typename S>
__device__ __forceinline__ float rest_of(int d, const CollideParams& p) {
    return Storage<S>::deviation ? (is_face(d) ? p.wface : p.wedge) : 0.f;
}

struct Quad {
    int i, k, j0;     // cells (i, j0 .. j0+V-1, k)
    int row;          // i*nz + k
    int e0;           // element index of (row, j0)
    bool active;      // j0 < ny (the quad holds at least one cell)
};

// MUL_DIV: divide by multiply-high (Dims::by_nq, by_nz). Measured on B200
// at 400^3: 5 % faster for the 16-bit kernels (issue-bound), but 4-11 %
// slower for the FP32 ones, whose loads the compiler then schedules worse;
// the FP32 kernels keep the hardware division sequence.
template <int V, bool MUL_DIV>
__device__ __forceinline__ Quad quad_of(const Dims& g, int nq, unsigned t) {
    Quad q;
    const unsigned total = (unsigned)g.nx * (unsigned)g.nz * (unsigned)nq;
    const unsigned tc = t < total ? t : total - 1;   // keep spare lanes on a valid quad
    static_assert(V == 1 || V == 2 || V == 4, "cells per thread");
    unsigned row;
    if (MUL_DIV) {
        row = g.by_nq[V >> 1].div(tc);   // V = 1, 2, 4: entries 0, 1, 2
        q.i = (int)g.by_nz.div(row);
    } else {
        row = tc / (unsigned)nq;
        q.i = (int)(row / (unsigned)g.nz);
    }
    const int jq = (int)(tc - row * (unsigned)nq);
    q.row = (int)row;
    q.k = (int)row - q.i * g.nz;
    q.j0 = jq * V;
    q.e0 = (int)row * g.jp + q.j0;
    q.active = t < total && q.j0 < g.ny;
    return q;
}

// The number of a launch's thread: its quad (parts 0 and 1) or its word of the list.
template <int V, int PART>
__device__ __forceinline__ unsigned part_number() {
    return PART == 2 ? listed_word(blockIdx.x, threadIdx.x, V) : blockIdx.x * blockDim.x + threadIdx.x;
}

// The quad of thread t of a launch (StepPart) and, per cell, whether this launch
// stores it (ok, V bits). PART 2: SEG = 32 / V consecutive lanes share a word of
// the list; lanes past the row's end take its last quad, inactive.
template <int V, bool MUL_DIV, int PART>
__device__ __forceinline__ Quad part_quad(const Dims& g, const StepPart& part, unsigned t, unsigned& ok) {
    constexpr unsigned ALL = (1u << V) - 1u;
    if constexpr (PART != 2) {
        const Quad q = quad_of<V, MUL_DIV>(g, g.jp / V, t);
        ok = q.active ? ALL : 0u;
        if constexpr (PART == 1)
            if (__ldg(part.skip + (size_t)q.row * g.jw + (q.j0 >> 5))) ok = 0u;
        return q;
    } else {
        constexpr unsigned SEG = 32 / V;
        const unsigned in = min(t, (unsigned)part.count - 1u);
        const int wd = part.words ? __ldg(part.words + in) : (int)in;
        const unsigned ex = part.except ? __ldg(part.except + wd) : 0u;
        Quad q;
        q.row = wd / g.jw;
        const int j = (wd - q.row * g.jw) * 32 + (int)(threadIdx.x % SEG) * V;
        q.i = q.row / g.nz;
        q.k = q.row - q.i * g.nz;
        q.j0 = min(j, g.jp - V);
        q.e0 = q.row * g.jp + q.j0;
        q.active = t < (unsigned)part.count && j < g.ny;
        unsigned live = 0u;
#pragma unroll
        for (int e = 0; e < V; e++) live |= j + e < g.ny ? 1u << e : 0u;
        ok = q.active ? live & ~(ex >> (j & 31)) : 0u;
        return q;
    }
}

// FORCE = false: the cells are known to lie outside every immersed-boundary
// stencil (the outer part of a split step), so F is zero without reading the
// touched flags.
template <int V, bool LES, bool COLLIDE, bool DEV, bool FORCE = true, bool FAST = false>
__device__ __forceinline__ void collide_quad(float (&f)[NQ][V], const Quad& q, float* __restrict__ Nu,
                                             const float4* __restrict__ F, const uint32_t* __restrict__ mask,
                                             const Dims& g, const CollideParams& p, bool from_moments, float (&nu)[V]) {
    if (!COLLIDE) return;
    float fx[V], fy[V], fz[V];
    const uint32_t bits =
        FORCE ? (__ldg(mask + (size_t)q.row * g.jw + (q.j0 >> 5)) >> (q.j0 & 31)) & ((1u << V) - 1u) : 0u;
    if (bits) {
#pragma unroll
        for (int e = 0; e < V; e++) {
            const float4 v = F[q.e0 + e];
            fx[e] = v.x;
            fy[e] = v.y;
            fz[e] = v.z;
        }
#pragma unroll
        for (int e = 0; e < V; e++)
            if (!((bits >> e) & 1u)) fx[e] = fy[e] = fz[e] = 0.f;
    } else {
#pragma unroll
        for (int e = 0; e < V; e++) fx[e] = fy[e] = fz[e] = 0.f;
    }
    if (LES) vload<V>(Nu + q.e0, nu);
    if constexpr (DEV && V >= 2) {
        // 16-bit storage, several cells per thread: two cells at a time in
        // packed FP32x2 arithmetic (the state always holds populations)
#pragma unroll
        for (int e = 0; e < V; e += 2) {
            F2 qv[NQ], m[NQ];
#pragma unroll
            for (int d = 0; d < NQ; d++) qv[d] = f2(f[d][e], f[d][e + 1]);
            moments_of(qv, m);
            F2 n = LES ? f2(nu[e], nu[e + 1]) : f2(0.f);
            collide<LES, DEV, FAST>(m, f2(fx[e], fx[e + 1]), f2(fy[e], fy[e + 1]), f2(fz[e], fz[e + 1]), n, p, qv);
            if (LES) {
                nu[e] = n.v.x;
                nu[e + 1] = n.v.y;
            }
#pragma unroll
            for (int d = 0; d < NQ; d++) {
                f[d][e] = qv[d].v.x;
                f[d][e + 1] = qv[d].v.y;
            }
        }
    } else {
#pragma unroll
        for (int e = 0; e < V; e++) {
            float qv[NQ], m[NQ];
#pragma unroll
            for (int d = 0; d < NQ; d++) qv[d] = f[d][e];
            if (from_moments) {
#pragma unroll
                for (int d = 0; d < NQ; d++) m[d] = qv[d];
            } else {
                moments_of(qv, m);
            }
            float n = LES ? nu[e] : 0.f;
            collide<LES, DEV, FAST>(m, fx[e], fy[e], fz[e], n, p, qv);
            if (LES) nu[e] = n;
#pragma unroll
            for (int d = 0; d < NQ; d++) f[d][e] = qv[d];
        }
    }
}

// ---------------------------------------------------------------------------
// Residual box (16-bit storage; tdlb::ResidualBox). A step with a box steps the
// cells of a list with k_box_step: with the residuals of their locations
// added on reading and kept on writing. The other launches of the step leave
// those cells out (StepPart::except): a cell's locations are its own alone,
// so the launches do not meet. f holds the cell's 18 values in direction
// order. The 18 residual loads leave together (a location outside the box reads
// the first residual instead): behind a branch each, they came one trip to the
// L2 after the other.
// ---------------------------------------------------------------------------
// Simple: add the residuals of the source locations inside the box (x - c_d,
// or the cell itself where x - c_d is off the lattice).
__device__ __forceinline__ void box_pull_simple(const ResidualBox& rr, int i, int j, int k, const Dims& g,
                                                float (&f)[NQ][1]) {
    float v[NQ];
    bool on[NQ];
#pragma unroll
    for (int d = 0; d < NQ; d++) {
        const int si = i - cx_of(d), sj = j - cy_of(d), sk = k - cz_of(d);
        const bool in = (unsigned)si < (unsigned)g.nx && (unsigned)sj < (unsigned)g.ny && (unsigned)sk < (unsigned)g.nz;
        const int li = in ? si : i, lj = in ? sj : j, lk = in ? sk : k;
        on[d] = rr.contains(li, lj, lk);
        v[d] = *(on[d] ? rr.at(d, li, lj, lk) : rr.res);
    }
#pragma unroll
    for (int d = 0; d < NQ; d++)
        if (on[d]) f[d][0] += v[d];
}
// Esotwist: slot s of cell (i, j, k) lives at (li, lj, lk); on reading, it
// holds direction EVEN ? s : s ^ 1, on writing EVEN ? s ^ 1 : s.
template <bool EVEN>
__device__ __forceinline__ void eso_location(int s, int i, int j, int k, int i1, int j1, int k1, int& li, int& lj,
                                             int& lk) {
    const int sg = EVEN ? -1 : 1;
    li = sg * cx_of(s) > 0 ? i1 : i;
    lj = sg * cy_of(s) > 0 ? j1 : j;
    lk = sg * cz_of(s) > 0 ? k1 : k;
}
template <bool EVEN>
__device__ __forceinline__ void box_read_eso(const ResidualBox& rb, int i, int j, int k, int i1, int j1, int k1,
                                             float (&f)[NQ][1]) {
    float v[NQ];
    bool on[NQ];
#pragma unroll
    for (int s = 0; s < NQ; s++) {
        int li, lj, lk;
        eso_location<EVEN>(s, i, j, k, i1, j1, k1, li, lj, lk);
        on[s] = rb.contains(li, lj, lk);
        v[s] = *(on[s] ? rb.at(s, li, lj, lk) : rb.res);
    }
#pragma unroll
    for (int s = 0; s < NQ; s++)
        if (on[s]) f[EVEN ? s : (s ^ 1)][0] += v[s];
}
// ---------------------------------------------------------------------------
// Simple (A/B, pull).
//
// All loads of a thread are issued as one straight-line batch (no branch
// between them), so the 18 population fetches of a quad are in flight
// together. V = 1 pulls every population directly from x - c_d. V > 1 loads
// aligned vectors of the upstream rows and moves j-shifted values between
// lanes with shuffles; the values a lane cannot get from a neighbour (warp
// edges) and the own values the wall rule needs at row ends come from scalar
// loads of those lanes alone, issued in the same batch. (Issued by every lane,
// as they were, they doubled the load instructions of the 16-bit kernels.)
// ---------------------------------------------------------------------------
template <typename S, int V, bool LES, bool FROM_MOMENTS, bool COLLIDE, int PART = 0>
__device__ __forceinline__ void simple_quad(const Planes& A, const Planes& B, float* __restrict__ Nu,
                                            const float4* __restrict__ F, const uint32_t* __restrict__ mask,
                                            const Dims& g, const CollideParams& p, unsigned t,
                                            const StepPart& part = StepPart{}) {
    static_assert(!(Storage<S>::deviation && FROM_MOMENTS), "16-bit state always holds populations");
    constexpr int SEG = PART == 2 ? 32 / V : 32;   // lanes that hold consecutive quads
    constexpr unsigned ALL = (1u << V) - 1u;
    unsigned ok;
    const Quad q = part_quad<V, sizeof(S) == 2, PART>(g, part, t, ok);
    const int lane = threadIdx.x & (SEG - 1);
    const int rs = g.nz * g.jp;   // elements per i step
    const bool i_lo = q.i == 0, i_hi = q.i == g.nx - 1, k_lo = q.k == 0, k_hi = q.k == g.nz - 1;
    const bool j_first = q.j0 == 0, j_last = q.j0 + V >= g.ny;
    float f[NQ][V];
    if (FROM_MOMENTS) {
#pragma unroll
        for (int d = 0; d < NQ; d++) pload<S, V, true>(A.p[d], q.e0, f[d]);
    } else if (V == 1) {
        // direct (unaligned) read-only loads: the texture path serves the
        // j-shifted rows better here than aligned loads plus lane shuffles
#pragma unroll
        for (int d = 0; d < NQ; d++) {
            const int cx = cx_of(d), cy = cy_of(d), cz = cz_of(d);
            // upstream cell x - c_d; off the lattice -> the cell keeps its own value
            const bool in = !((cx > 0 && i_lo) || (cx < 0 && i_hi) || (cz > 0 && k_lo) || (cz < 0 && k_hi) ||
                              (cy > 0 && j_first) || (cy < 0 && j_last));
            const int off = in ? -(cx * rs + cz * g.jp + cy) : 0;
            f[d][0] = pload1<S, true>(A.p[d], q.e0 + off);
        }
    } else {
        float ext[NQ];   // what a lane cannot get from its neighbour
        // batch 1: every load
#pragma unroll
        for (int d = 0; d < NQ; d++) {
            const int cx = cx_of(d), cy = cy_of(d), cz = cz_of(d);
            const bool row_ok = !((cx > 0 && i_lo) || (cx < 0 && i_hi) || (cz > 0 && k_lo) || (cz < 0 && k_hi));
            const int soff = row_ok ? -(cx * rs + cz * g.jp) : 0;
            const int src = q.e0 + soff;
            pload<S, V, true>(A.p[d], src, f[d]);
            if (cy > 0) {
                ext[d] = (j_first || lane == 0) ? pload1<S, true>(A.p[d], j_first ? q.e0 : src - 1) : 0.f;
            } else if (cy < 0) {
                int le = g.ny - 1 - q.j0;
                le = le < 0 ? 0 : (le > V - 1 ? V - 1 : le);
                ext[d] = (j_last || lane == SEG - 1) ? pload1<S, true>(A.p[d], j_last ? q.e0 + le : src + V) : 0.f;
            }
        }
        // batch 2: shift along j
#pragma unroll
        for (int d = 0; d < NQ; d++) {
            const int cx = cx_of(d), cy = cy_of(d), cz = cz_of(d);
            const bool row_ok = !((cx > 0 && i_lo) || (cx < 0 && i_hi) || (cz > 0 && k_lo) || (cz < 0 && k_hi));
            if (cy > 0) {                          // source j - 1
                const float left = __shfl_up_sync(FULL, f[d][V - 1], 1);
                if (row_ok) {
#pragma unroll
                    for (int e = V - 1; e > 0; e--) f[d][e] = f[d][e - 1];
                    f[d][0] = (j_first || lane == 0) ? ext[d] : left;
                }
            } else if (cy < 0) {                   // source j + 1
                const float right = __shfl_down_sync(FULL, f[d][0], 1);
                const int le = g.ny - 1 - q.j0;   // element of the row's last cell when j_last
                if (row_ok) {
#pragma unroll
                    for (int e = 0; e < V - 1; e++) f[d][e] = f[d][e + 1];
                    f[d][V - 1] = lane == SEG - 1 ? ext[d] : right;
                    if (j_last) {
#pragma unroll
                        for (int e = 0; e < V; e++)
                            if (e == le) f[d][e] = ext[d];
                    }
                }
            }
        }
    }
    float nu[V];
    // 16-bit storage: approximate reciprocals and square root (measured on
    // B200 at 400^3: FP16 step 1.28 -> 1.19 ms; the Esotwist kernel, which
    // keeps IEEE rounding, measured slower with them, 1.38 -> 1.47 ms)
    collide_quad<V, LES, COLLIDE, Storage<S>::deviation, PART != 1, Storage<S>::deviation>(f, q, Nu, F, mask, g,
                                                                                           p, FROM_MOMENTS, nu);
    if (!ok) return;
    if (PART == 2 && ok != ALL) {
#pragma unroll
        for (int e = 0; e < V; e++) {
            if (!((ok >> e) & 1u)) continue;
#pragma unroll
            for (int d = 0; d < NQ; d++) pstore1<S>(B.p[d], q.e0 + e, f[d][e]);
            if (COLLIDE && LES) Nu[q.e0 + e] = nu[e];
        }
        return;
    }
#pragma unroll
    for (int d = 0; d < NQ; d++) pstore<S, V, sizeof(S) == 4>(B.p[d], q.e0, f[d]);
    if constexpr (sizeof(S) == 4) {
        if (COLLIDE && LES) vstore_cs<V>(Nu + q.e0, nu);
    } else {
        if (COLLIDE && LES) vstore<V>(Nu + q.e0, nu);
    }
}

// ---------------------------------------------------------------------------
// Esotwist (single buffer, in place).
//
// Slot s of cell x lives at x + o_s, o_s = max(-c_s, 0) (even) or
// max(+c_s, 0) (odd), +1 wrapping to 0; a cell reads and writes the same 18
// locations. V = 1 addresses them directly. For V > 1, where o_s has a j
// component the V locations of a quad are j0+1 .. j0+V: loads take the
// aligned vector at j0 and the next lane's first element; stores write the
// aligned vector at j0 holding the previous lane's last value, and the lane
// that owns the last cell of a warp (or of a row, where the location wraps to
// j = 0) stores that one value alone. A __syncwarp() separates every lane's
// loads from any lane's stores, so a location is always read by its owner
// before a neighbour overwrites it.
// ---------------------------------------------------------------------------
template <typename S, int V, bool LES, bool FROM_MOMENTS, bool COLLIDE, bool EVEN, int PART = 0>
__device__ __forceinline__ void esotwist_quad(const Planes& Q, float* __restrict__ Nu, const float4* __restrict__ F,
                                              const uint32_t* __restrict__ mask, const Dims& g, const CollideParams& p,
                                              unsigned t, const StepPart& part = StepPart{}) {
    static_assert(!(Storage<S>::deviation && FROM_MOMENTS), "16-bit state always holds populations");
    constexpr int SEG = PART == 2 ? 32 / V : 32;   // lanes that hold consecutive quads
    constexpr unsigned ALL = (1u << V) - 1u;
    unsigned ok_cells;
    const Quad q = part_quad<V, sizeof(S) == 2, PART>(g, part, t, ok_cells);
    const int lane = threadIdx.x & (SEG - 1);
    const int i1 = q.i + 1 == g.nx ? 0 : q.i + 1;
    const int k1 = q.k + 1 == g.nz ? 0 : q.k + 1;
    const bool j_last = q.j0 + V >= g.ny;
    const int last_e = g.ny - 1 - q.j0;   // element holding the row's last cell (if < V)
    float f[NQ][V];
    if (V == 1) {
        // Slots with a j offset read element j + 1: every lane loads its own
        // (aligned) element j and takes j + 1 from the next lane; the lane at
        // a warp's end or a row's end loads its element itself. (Padding
        // lanes, j >= ny, load element 0 of their row: in bounds, unused.)
        const bool row_end = q.j0 == g.ny - 1;
        const bool warp_end = lane == 31;
        const int j1 = (row_end || q.j0 >= g.ny) ? 0 : q.j0 + 1;
        float v[NQ], x[NQ];
#pragma unroll
        for (int s = 0; s < NQ; s++) {
            const int sg = EVEN ? -1 : 1;
            const bool oi = sg * cx_of(s) > 0, oj = sg * cy_of(s) > 0, ok = sg * cz_of(s) > 0;
            const int base = ((oi ? i1 : q.i) * g.nz + (ok ? k1 : q.k)) * g.jp;
            v[s] = pload1<S, false>(Q.p[s], base + q.j0);
            if (oj) x[s] = (warp_end || row_end) ? pload1<S, false>(Q.p[s], base + j1) : 0.f;
        }
#pragma unroll
        for (int s = 0; s < NQ; s++) {
            const int sg = EVEN ? -1 : 1;
            const bool oj = sg * cy_of(s) > 0;
            const int d = EVEN ? s : (s ^ 1);
            if (oj) {
                const float right = __shfl_down_sync(FULL, v[s], 1);
                f[d][0] = (warp_end || row_end) ? x[s] : right;
            } else {
                f[d][0] = v[s];
            }
        }
    } else {
        float ext[NQ];   // what a lane cannot get from the next one
#pragma unroll
        for (int s = 0; s < NQ; s++) {
            const int sg = EVEN ? -1 : 1;
            const bool oi = sg * cx_of(s) > 0, oj = sg * cy_of(s) > 0, ok = sg * cz_of(s) > 0;
            const int d = EVEN ? s : (s ^ 1);
            const int base = ((oi ? i1 : q.i) * g.nz + (ok ? k1 : q.k)) * g.jp;
            pload<S, V, false>(Q.p[s], base + q.j0, f[d]);
            if (oj) {
                ext[s] = (j_last || lane == SEG - 1) ? pload1<S, false>(Q.p[s], base + (j_last ? 0 : q.j0 + V)) : 0.f;
            }
        }
#pragma unroll
        for (int s = 0; s < NQ; s++) {
            const int sg = EVEN ? -1 : 1;
            const bool oj = sg * cy_of(s) > 0;
            const int d = EVEN ? s : (s ^ 1);
            if (!oj) continue;
            const float right = __shfl_down_sync(FULL, f[d][0], 1);
#pragma unroll
            for (int e = 0; e < V - 1; e++) f[d][e] = f[d][e + 1];
            f[d][V - 1] = lane == SEG - 1 ? ext[s] : right;
            if (j_last) {                          // j = ny-1 wraps to 0
#pragma unroll
                for (int e = 0; e < V; e++)
                    if (e == last_e) f[d][e] = ext[s];
            }
        }
    }
    __syncwarp();
    float nu[V];
    collide_quad<V, LES, COLLIDE, Storage<S>::deviation, PART != 1>(f, q, Nu, F, mask, g, p, FROM_MOMENTS, nu);
    // A location of the next cell along j is written by the next lane: bit e of
    // put: this launch stores the cell before element e.
    unsigned put = ALL;
    if constexpr (PART != 0) put = (__shfl_up_sync(FULL, ok_cells, 1) >> (V - 1)) | (ok_cells << 1);
    if (V == 1) {
        // Slots with a j offset write element j + 1: lane l writes element j
        // with the value of the previous lane (cell j - 1, same row), so the
        // warp's store is aligned; the lane at a warp's end or a row's end
        // writes its own element j + 1 (j = ny - 1: element 0) itself.
        const bool row_end = q.j0 == g.ny - 1;
        const bool warp_end = lane == 31;
        const int j1 = (row_end || q.j0 >= g.ny) ? 0 : q.j0 + 1;
#pragma unroll
        for (int s = 0; s < NQ; s++) {
            const int sg = EVEN ? -1 : 1;
            const bool oi = sg * cx_of(s) > 0, oj = sg * cy_of(s) > 0, ok = sg * cz_of(s) > 0;
            const int d = EVEN ? (s ^ 1) : s;
            const int base = ((oi ? i1 : q.i) * g.nz + (ok ? k1 : q.k)) * g.jp;
            if (!oj) {
                if (ok_cells) pstore1<S>(Q.p[s], base + q.j0, f[d][0]);
                continue;
            }
            const float left = __shfl_up_sync(FULL, f[d][0], 1);
            if (lane > 0 && q.j0 > 0 && q.j0 <= g.ny - 1 && q.active && (put & 1u))
                pstore1<S>(Q.p[s], base + q.j0, left);
            if (ok_cells && (warp_end || row_end)) pstore1<S>(Q.p[s], base + j1, f[d][0]);
        }
        if (COLLIDE && LES && ok_cells) Nu[q.e0] = nu[0];
        return;
    }
    const bool j_first = q.j0 == 0;
#pragma unroll
    for (int s = 0; s < NQ; s++) {
        const int sg = EVEN ? -1 : 1;
        const bool oi = sg * cx_of(s) > 0, oj = sg * cy_of(s) > 0, ok = sg * cz_of(s) > 0;
        const int d = EVEN ? (s ^ 1) : s;      // direction written to slot s
        const int base = ((oi ? i1 : q.i) * g.nz + (ok ? k1 : q.k)) * g.jp;
        if (!oj) {
            if (PART == 2 && ok_cells != ALL) {
#pragma unroll
                for (int e = 0; e < V; e++)
                    if ((ok_cells >> e) & 1u) pstore1<S>(Q.p[s], base + q.j0 + e, f[d][e]);
            } else if (ok_cells) {
                pstore<S, V>(Q.p[s], base + q.j0, f[d]);
            }
            continue;
        }
        float w[V];
        const float prev = __shfl_up_sync(FULL, f[d][V - 1], 1);
        w[0] = prev;
#pragma unroll
        for (int e = 1; e < V; e++) w[e] = f[d][e - 1];
        if (!q.active) continue;
        if (lane != 0 && !j_first && (PART == 0 || (put & ALL) == ALL)) {
            pstore<S, V>(Q.p[s], base + q.j0, w);
        } else {
            if (PART != 0 && lane != 0 && !j_first && (put & 1u)) pstore1<S>(Q.p[s], base + q.j0, w[0]);
#pragma unroll
            for (int e = 1; e < V; e++)
                if (PART == 0 || ((put >> e) & 1u)) pstore1<S>(Q.p[s], base + q.j0 + e, w[e]);
        }
        if (j_last) {                          // the wrap location of j = ny-1
#pragma unroll
            for (int e = 0; e < V; e++)
                if (e == last_e && (PART == 0 || ((ok_cells >> e) & 1u))) pstore1<S>(Q.p[s], base, f[d][e]);
        } else if (lane == SEG - 1 && (PART == 0 || ((ok_cells >> (V - 1)) & 1u))) {
            pstore1<S>(Q.p[s], base + q.j0 + V, f[d][V - 1]);
        }
    }
    if (COLLIDE && LES && ok_cells) {
        if (PART == 2 && ok_cells != ALL) {
#pragma unroll
            for (int e = 0; e < V; e++)
                if ((ok_cells >> e) & 1u) Nu[q.e0 + e] = nu[e];
        } else {
            vstore<V>(Nu + q.e0, nu);
        }
    }
}


// Split step. The immersed-boundary pass of a step touches a thin set of
// cells, so a step can run as two launches over the flag words (StepPart):
//   PART 1 (outer): the words outside the zone; F is zero there, so this
//     launch reads neither F nor the touched flags. It walks the whole lattice
//     as PART 0 does, prefetch included, and drops the zone's results at the
//     store (a few per cent of the cells): the flag is loaded beside the
//     populations and delays nothing;
//   PART 2 (inner): the words of the zone, from a list, or, for a step with a
//     residual box and no zone, every word.
// PART 0 runs every cell. The outer launch of a step depends on the previous
// step's populations only, so it can run while the previous forcing pass is
// still in flight.
// L2 prefetch ahead of a full launch's walk. CTA b covers elements
// [128 V b, 128 V (b + 1)) of the flat row * jp + j index. Every
// kPrefetchTiles-th CTA, as it starts, has NQ + 1 of its threads issue one
// cp.async.bulk.prefetch.L2 each, for the kPrefetchTiles tiles that begin
// `ahead` CTAs later: the span of plane d the pull reads (Simple: the tiles
// shifted by -c_d; Esotwist: shifted to the row of slot d's location) and
// Nu's span (LES). With `ahead` one wave of resident CTAs, the populations
// are in L2 when those CTAs load them, so the loads -- whose latency bounds
// the kernels at their occupancy -- wait for the L2, not for the DRAM.
// Measured on B200 at 400^3 (step kernel alone, ms): FP32 Simple 1.558 ->
// 1.462, FP32 Esotwist 1.741 -> 1.483, 16-bit Simple (four cells per thread)
// 1.110 -> 0.905, 16-bit Esotwist (two cells per thread) 1.252 -> 1.081.
// Spans are clamped to the plane and rounded out to 16 bytes (planes start
// 16-byte aligned and hold a multiple of 64 elements); a prefetch changes no
// result.
constexpr int kPrefetchTiles = 8;
// What the cells of elements [e0, e1) read of population plane d (d == NQ: of Nu,
// their own elements), as bytes from the plane's base; empty where lo >= hi.
struct PrefetchSpan {
    long long lo, hi;
};
__host__ __device__ __forceinline__ PrefetchSpan pull_span(const Dims& g, int d, int es, bool eso, bool even, long long e0,
                                                           long long e1) {
    if (d < NQ) {
        const long long rs = (long long)g.nz * g.jp;
        long long sh;
        if (eso) {
            const int sg = even ? -1 : 1;
            sh = (sg * cx_of(d) > 0 ? rs : 0) + (sg * cz_of(d) > 0 ? g.jp : 0);
        } else {
            sh = -(cx_of(d) * rs + cz_of(d) * g.jp);
        }
        // one element either side: the j +- 1 neighbours
        e0 += sh - 1;
        e1 += sh + 1;
    }
    e0 = e0 < 0 ? 0 : e0;
    e1 = e1 > g.plane ? g.plane : e1;
    if (e0 >= e1) return PrefetchSpan{0, 0};
    return PrefetchSpan{e0 * es & ~15LL, (e1 * es + 15) & ~15LL};
}
__device__ __forceinline__ void prefetch_span(const void* base, PrefetchSpan s) {
    if (s.lo >= s.hi) return;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"((const char*)base + s.lo), "r"((unsigned)(s.hi - s.lo))
                 : "memory");
}
template <typename S, int V, bool LES, bool ESO, bool EVEN>
__device__ __forceinline__ void prefetch_ahead(const Planes& A, const float* Nu, const Dims& g, int ahead) {
    const int d = (int)threadIdx.x;
    if (ahead <= 0 || d >= (LES ? NQ + 1 : NQ) || blockIdx.x % kPrefetchTiles) return;
    constexpr long long tile = 128LL * V;
    const long long e0 = ((long long)blockIdx.x + ahead) * tile, e1 = e0 + kPrefetchTiles * tile;
    if (e0 >= g.rows() * g.jp) return;
    // (two calls: with the plane chosen by a select, the 16-bit Esotwist kernel's outer
    // launch is slower, 400^3 FP16 whole step 1.498 -> 1.532 ms)
    if (d == NQ) return prefetch_span(Nu, pull_span(g, NQ, 4, ESO, EVEN, e0, e1));
    prefetch_span(A.p[d], pull_span(g, d, (int)sizeof(S), ESO, EVEN, e0, e1));
}

// Step launches that go close behind the one before them (launch_chained): all
// but part 1, which follows an event on a stream of its own.
template <int PART>
constexpr bool kChained = PART != 1;

template <typename S, int V, bool LES, bool FROM_MOMENTS, bool COLLIDE, int PART = 0>
__global__ void __launch_bounds__(128, 4) k_step_simple(Planes A, Planes B, float* __restrict__ Nu,
                                                       const float4* __restrict__ F, const uint32_t* __restrict__ mask,
                                                       Dims g, CollideParams p, StepPart part) {
    if constexpr (PART != 2 && COLLIDE && !FROM_MOMENTS)
        prefetch_ahead<S, V, LES, false, false>(A, Nu, g, part.l2_ahead);
    unsigned t = part_number<V, PART>();
    if constexpr (kChained<PART>) after_previous(t);
    simple_quad<S, V, LES, FROM_MOMENTS, COLLIDE, PART>(A, B, Nu, F, mask, g, p, t, part);
}

// Resident 128-thread blocks per SM the Esotwist kernel is built for: the
// register cap that follows (64 at one cell per thread) keeps enough loads in
// flight; measured on B200 at 400^3, 8 blocks beat 4 by about 5%. 16-bit storage
// at two cells per thread: 5 blocks 1.287 ms, 6 1.127, 7 1.100, 8 1.071; at four:
// 3 1.420, 4 1.150, 5 1.183, 6 1.274.
template <typename S, int V>
constexpr int kEsotwistBlocksPerSM = V == 1 ? 8 : V == 2 ? (sizeof(S) == 2 ? 8 : 6) : 4;

template <typename S, int V, bool LES, bool FROM_MOMENTS, bool COLLIDE, bool EVEN, int PART = 0>
__global__ void __launch_bounds__(128, kEsotwistBlocksPerSM<S, V>) k_step_esotwist(Planes Q, float* __restrict__ Nu,
                                                         const float4* __restrict__ F, const uint32_t* __restrict__ mask,
                                                         Dims g, CollideParams p, StepPart part) {
    if constexpr (PART != 2 && COLLIDE && !FROM_MOMENTS)
        prefetch_ahead<S, V, LES, true, EVEN>(Q, Nu, g, part.l2_ahead);
    unsigned t = part_number<V, PART>();
    if constexpr (kChained<PART>) after_previous(t);
    esotwist_quad<S, V, LES, FROM_MOMENTS, COLLIDE, EVEN, PART>(Q, Nu, F, mask, g, p, t, part);
}

template <bool CHAINED, typename... P, typename... A>
cudaError_t launch_step_kernel(void (*kernel)(P...), unsigned grid, cudaStream_t st, A... args) {
    if constexpr (CHAINED) {
        return launch_chained(kernel, grid, 128, 0, st, args...);
    } else {
        kernel<<<grid, 128, 0, st>>>(static_cast<P>(args)...);
        return cudaGetLastError();
    }
}

// One cell of the box list per thread: its 18 stored deviations, exact where
// their locations lie in the box (rr), collided as the one-cell-per-thread
// step kernels do and written with the residuals of the locations inside the
// box (rw: the destination's set, the same one for Esotwist). Scattered runs of
// a few tens of cells: bound by load latency (B200, beside the outer words: 160^3
// FP16 Simple 20 us, 400^3 FP16 Esotwist 114; stepping into a scratch array and
// committing it afterwards took 27.5 and 136).
template <typename S, bool SIMPLE, bool LES, bool EVEN>
__global__ void __launch_bounds__(128) k_box_step(Planes A, Planes B, float* __restrict__ Nu, const float4* __restrict__ F,
                                                  const uint32_t* __restrict__ mask, Dims g, CollideParams p,
                                                  const int* __restrict__ cells, int n, ResidualBox rr, ResidualBox rw) {
    int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    after_previous(t);
    if (t >= n) return;
    Quad q;
    q.e0 = cells[t];
    q.row = q.e0 / g.jp;
    q.j0 = q.e0 - q.row * g.jp;
    q.i = q.row / g.nz;
    q.k = q.row - q.i * g.nz;
    q.active = true;
    const int i1 = q.i + 1 == g.nx ? 0 : q.i + 1, j1 = q.j0 + 1 == g.ny ? 0 : q.j0 + 1, k1 = q.k + 1 == g.nz ? 0 : q.k + 1;
    float f[NQ][1];
#pragma unroll
    for (int s = 0; s < NQ; s++) {
        if constexpr (SIMPLE) {
            const int si = q.i - cx_of(s), sj = q.j0 - cy_of(s), sk = q.k - cz_of(s);
            const bool in = (unsigned)si < (unsigned)g.nx && (unsigned)sj < (unsigned)g.ny && (unsigned)sk < (unsigned)g.nz;
            f[s][0] = pload1<S, false>(A.p[s], in ? (int)g.at(si, sj, sk) : q.e0);
        } else {
            int li, lj, lk;
            eso_location<EVEN>(s, q.i, q.j0, q.k, i1, j1, k1, li, lj, lk);
            f[EVEN ? s : (s ^ 1)][0] = pload1<S, false>(A.p[s], (int)g.at(li, lj, lk));
        }
    }
    if (rr.near(q.i, q.j0, q.k)) {
        if constexpr (SIMPLE) box_pull_simple(rr, q.i, q.j0, q.k, g, f);
        else box_read_eso<EVEN>(rr, q.i, q.j0, q.k, i1, j1, k1, f);
    }
    float nu[1];
    collide_quad<1, LES, true, true, true, SIMPLE>(f, q, Nu, F, mask, g, p, false, nu);
#pragma unroll
    for (int s = 0; s < NQ; s++) {
        int li = q.i, lj = q.j0, lk = q.k;
        if (!SIMPLE) eso_location<EVEN>(s, q.i, q.j0, q.k, i1, j1, k1, li, lj, lk);
        const float v = f[SIMPLE ? s : (EVEN ? (s ^ 1) : s)][0];
        const S enc = Storage<S>::enc(v);
        reinterpret_cast<S*>((SIMPLE ? B : A).p[s])[g.at(li, lj, lk)] = enc;
        if (rw.contains(li, lj, lk)) *rw.at(s, li, lj, lk) = v - Storage<S>::dec(enc);
    }
    if (LES) Nu[q.e0] = nu[0];
}

// Moments of the current state at an interior cell (what the reference's Q
// holds after moments()). mode: 0 = Simple populations (pull), 1 = moments (own cell),
// 2 = Esotwist populations (read map, parity `even`), 3 = Esotwist moments.
template <typename S>
__device__ __forceinline__ void state_moments18(const Planes& A, const Dims& g, int mode, int even, const CollideParams& p,
                                                int i, int j, int k, float (&m)[NQ],
                                                const ResidualBox rb = ResidualBox{}) {
    const int e = (int)g.at(i, j, k);
    float q[NQ];
    if (mode <= 1) {
#pragma unroll
        for (int d = 0; d < NQ; d++) {
            int src = e;
            if (mode == 0) {
                const int si = i - cx_of(d), sj = j - cy_of(d), sk = k - cz_of(d);
                const bool in = (unsigned)si < (unsigned)g.nx && (unsigned)sj < (unsigned)g.ny && (unsigned)sk < (unsigned)g.nz;
                if (in) src = (int)g.at(si, sj, sk);
                if (Storage<S>::deviation && rb.on()) {
                    const int li = in ? si : i, lj = in ? sj : j, lk = in ? sk : k;
                    if (rb.contains(li, lj, lk)) {
                        q[d] = pload1<S, false>(A.p[d], src) + *rb.at(d, li, lj, lk) + rest_of<S>(d, p);
                        continue;
                    }
                }
            }
            q[d] = pload1<S, false>(A.p[d], src) + (mode == 0 ? rest_of<S>(d, p) : 0.f);
        }
    } else {
        const int i1 = i + 1 == g.nx ? 0 : i + 1, j1 = j + 1 == g.ny ? 0 : j + 1, k1 = k + 1 == g.nz ? 0 : k + 1;
#pragma unroll
        for (int d = 0; d < NQ; d++) {
            const int s = even ? d : (d ^ 1);
            const int sg = even ? -1 : 1;
            const bool oi = sg * cx_of(s) > 0, oj = sg * cy_of(s) > 0, ok = sg * cz_of(s) > 0;
            q[d] = pload1<S, false>(A.p[s], (int)g.at(oi ? i1 : i, oj ? j1 : j, ok ? k1 : k)) +
                   (mode == 2 ? rest_of<S>(d, p) : 0.f);
            if (Storage<S>::deviation && mode == 2 && rb.on() && rb.contains(oi ? i1 : i, oj ? j1 : j, ok ? k1 : k))
                q[d] += *rb.at(s, oi ? i1 : i, oj ? j1 : j, ok ? k1 : k);
        }
    }
    if (mode == 0 || mode == 2) moments_of(q, m);
    else {
#pragma unroll
        for (int d = 0; d < NQ; d++) m[d] = q[d];
    }
}

}  // namespace tdlb
