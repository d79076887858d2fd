// The marker scheduler on the device: what MarkerSchedule and CellList
// (tdlb_runtime.hpp) make of the first segment of a marker list -- the order by
// (plane, level, list index), the levels, the unique stencil cells per plane
// with each marker's nine places among them, the touched flags -- from the list
// in device memory. The reference's main loop hands the whole list over with
// every step (main.cpp:409-454), so this is per-step work there. On the host it
// was one thread's pass over nine cells per marker, three times (144^3 tank,
// 75,000 markers: about 90 ms a call); here every plane is a block's and the
// list is read twice.
//
//   k_sched_count    (a warp per 256 or 1024 markers) range check, markers per
//                    plane
//   k_sched_offsets  per plane: running offsets over the chunks
//   k_sched_scan     plane offsets
//   k_sched_scatter  list indices by plane, in list order
//   k_sched_cells    (a block per plane) unique stencil cells: a bitmap
//   k_sched_levels   (a block per plane) places, levels, order
//   k_sched_finish   level offsets over the planes, then k_sched_level_ptr
//
// Levels: in each round the markers not yet placed write their index into
// their nine cells with atomicMin; a marker that finds its own in all nine has
// no earlier marker left to wait for. Round r so finds exactly the markers of
// level r = 1 + the highest level of an earlier marker sharing a cell. A round
// costs about 2 us for a plane of 1500 markers; a tank's wall has ten levels. A
// list with very long chains (thousands of markers on one cell) gives up after
// kMaxRounds and the host schedules it, whose time does not grow with the
// chains.
#include "tdlb_kernels.cuh"

#include <algorithm>

namespace tdlb {

constexpr int kSteps = 8;           // steps of 32 markers whose loads leave together
constexpr int kMaxRounds = 4096;
constexpr unsigned kAll = 0xffffffffu;
constexpr int kHeld = 3;           // markers of a plane a thread keeps in registers

__device__ __forceinline__ int marker_plane(const SchedArgs& a, int q) {
    const Marker& m = a.markers[q];
    const bool in = m.i >= 0 && m.i < a.g.nx && m.j >= 0 && m.j < a.g.ny && m.k >= 0 && m.k < a.g.nz;
    return in ? (int)m.j : -1;
}

// Markers of one warp, in list order: few, so that a short list is many warps
// (12,900 markers in warps of 1024 took 24 us a pass), more where the offsets of
// the chunks would be the longer pass.
static int chunk_of(long long n) { return n <= (1 << 17) ? 32 * kSteps : 128 * kSteps; }

__global__ void __launch_bounds__(128) k_sched_count(SchedArgs a, int nchunk, int per) {
    const int chunk = (int)(blockIdx.x * 4 + threadIdx.x / 32), lane = threadIdx.x & 31;
    if (chunk >= nchunk) return;
    for (int s = 0; s < per; s += 32 * kSteps) {
        const long long q0 = (long long)chunk * per + s + lane;
        int j[kSteps];
#pragma unroll
        for (int u = 0; u < kSteps; u++) {
            const long long q = q0 + 32 * u;
            j[u] = q < a.n ? marker_plane(a, (int)q) : -2;
        }
#pragma unroll
        for (int u = 0; u < kSteps; u++) {
            const long long q = q0 + 32 * u;
            if (j[u] == -1) atomicMin(a.info, (int)q);
            const int jj = q < a.n0 ? j[u] : -1;
            const unsigned same = __match_any_sync(kAll, jj);
            if (jj >= 0 && lane == __ffs(same) - 1) atomicAdd(a.hist + (long long)chunk * a.g.ny + jj, __popc(same));
        }
    }
}

// a warp per plane
__global__ void __launch_bounds__(128) k_sched_offsets(SchedArgs a, int nchunk) {
    const int j = (int)(blockIdx.x * 4 + threadIdx.x / 32), lane = threadIdx.x & 31;
    if (j >= a.g.ny) return;
    int sum = 0;
#pragma unroll 4
    for (int c0 = 0; c0 < nchunk; c0 += 32) {
        int* h = a.hist + (long long)(c0 + lane) * a.g.ny + j;
        const int v = c0 + lane < nchunk ? *h : 0;
        int s = v;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const int y = __shfl_up_sync(kAll, s, d);
            if (lane >= d) s += y;
        }
        if (c0 + lane < nchunk) *h = sum + s - v;
        sum += __shfl_sync(kAll, s, 31);
    }
    if (lane == 0) a.plane_slot[j] = sum;
}

// Exclusive scan of v[0, n) in place by one block of 1024 threads; v[n] = total.
__device__ __forceinline__ int block_scan(int* v, int n) {
    __shared__ int part[32];
    __shared__ int carry;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int b = 0; b < n; b += 1024) {
        const int t = b + (int)threadIdx.x;
        const int x = t < n ? v[t] : 0;
        int s = x;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const int y = __shfl_up_sync(kAll, s, d);
            if (lane >= d) s += y;
        }
        if (lane == 31) part[warp] = s;
        __syncthreads();
        if (warp == 0) {
            int p = part[lane];
#pragma unroll
            for (int d = 1; d < 32; d *= 2) {
                const int y = __shfl_up_sync(kAll, p, d);
                if (lane >= d) p += y;
            }
            part[lane] = p;
        }
        __syncthreads();
        const int before = carry + (warp ? part[warp - 1] : 0);
        if (t < n) v[t] = before + s - x;
        __syncthreads();
        if (threadIdx.x == 0) carry += part[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) v[n] = carry;
    return carry;
}

__global__ void __launch_bounds__(1024) k_sched_scan(SchedArgs a) { block_scan(a.plane_slot, a.g.ny); }

__global__ void __launch_bounds__(128) k_sched_scatter(SchedArgs a, int nchunk, int per) {
    const int chunk = (int)(blockIdx.x * 4 + threadIdx.x / 32), lane = threadIdx.x & 31;
    if (chunk >= nchunk) return;
    for (int s = 0; s < per; s += 32 * kSteps) {
        const long long q0 = (long long)chunk * per + s + lane;
        int j[kSteps], first[kSteps];
#pragma unroll
        for (int u = 0; u < kSteps; u++) {
            const long long q = q0 + 32 * u;
            j[u] = q < a.n0 ? marker_plane(a, (int)q) : -1;
        }
#pragma unroll
        for (int u = 0; u < kSteps; u++) first[u] = j[u] >= 0 ? a.plane_slot[j[u]] : 0;
#pragma unroll
        for (int u = 0; u < kSteps; u++) {
            const unsigned same = __match_any_sync(kAll, j[u]);
            const int leader = __ffs(same) - 1;
            int base = 0;
            if (j[u] >= 0 && lane == leader) base = atomicAdd(a.hist + (long long)chunk * a.g.ny + j[u], __popc(same));
            base = __shfl_sync(kAll, base, leader);
            if (j[u] >= 0) a.by_plane[first[u] + base + __popc(same & ((1u << lane) - 1u))] = (int)(q0 + 32 * u);
        }
    }
}

// The nine (i, k) cells of a marker's stencil as row numbers (Dims::row), in
// MarkerSchedule::stencil's order.
__device__ __forceinline__ void stencil_rows(const Marker& m, const Dims& g, int (&row)[9]) {
    int c = 0;
#pragma unroll
    for (int k1 = -1; k1 <= 1; k1++)
#pragma unroll
        for (int i1 = -1; i1 <= 1; i1++, c++) {
            int i = (int)m.i + i1, k = (int)m.k + k1;
            i = i < 0 ? i + g.nx : (i >= g.nx ? i - g.nx : i);
            k = k < 0 ? k + g.nz : (k >= g.nz ? k - g.nz : k);
            row[c] = (int)g.row(i, k);
        }
}

// A plane's bitmap of (i, k) cells: in shared memory, or, where an x * z plane
// does not fit, in the plane's part of a.maps.
__device__ __forceinline__ int map_words(const Dims& g) { return (int)((g.rows() + 31) / 32); }

template <int NT>
__device__ __forceinline__ void fill_map(const SchedArgs& a, int j, unsigned* map) {
    const int W = map_words(a.g), p0 = a.plane_slot[j], p1 = a.plane_slot[j + 1];
    for (int w = threadIdx.x; w < W; w += NT) map[w] = 0u;
    __syncthreads();
    for (int p = p0 + (int)threadIdx.x; p < p1; p += NT) {
        int row[9];
        stencil_rows(a.markers[a.by_plane[p]], a.g, row);
#pragma unroll
        for (int c = 0; c < 9; c++) atomicOr(map + (row[c] >> 5), 1u << (row[c] & 31));
    }
    __syncthreads();
}

__global__ void __launch_bounds__(256) k_sched_cells(SchedArgs a) {
    extern __shared__ unsigned smap[];
    __shared__ int total;
    const int j = (int)blockIdx.x, W = map_words(a.g);
    unsigned* map = a.maps ? a.maps + (size_t)j * 2 * W : smap;
    if (threadIdx.x == 0) total = 0;
    fill_map<256>(a, j, map);
    int n = 0;
    for (int w = threadIdx.x; w < W; w += 256) n += __popc(*(volatile unsigned*)(map + w));
    atomicAdd(&total, n);
    __syncthreads();
    if (threadIdx.x == 0) a.plane_count[j] = total;
}

// One block per plane. own_smem: the owner array (one int per cell of the plane)
// lies in shared memory behind the maps, else in a.owner.
template <int NT>
__global__ void __launch_bounds__(NT) k_sched_levels(SchedArgs a, int owner_cap) {
    extern __shared__ unsigned smap[];
    __shared__ int warps[NT / 32], counts[kHeld][NT / 32];
    __shared__ int placed;
    const int j = (int)blockIdx.x, W = map_words(a.g), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int p0 = a.plane_slot[j], m = a.plane_slot[j + 1] - p0, c0 = a.plane_cell[j], nc = a.plane_cell[j + 1] - c0;
    if (m == 0) {
        if (threadIdx.x == 0) a.levels[j] = 0;
        return;
    }
    unsigned* map = a.maps ? a.maps + (size_t)j * 2 * W : smap;
    int* pre = (int*)(map + W);   // cells before each word
    int* owner = nc <= owner_cap ? (int*)(a.maps ? smap : smap + 2 * W) : a.owner + c0;
    fill_map<NT>(a, j, map);
    // running cell numbers: each thread a run of words
    const int run = (W + NT - 1) / NT, w0 = min(W, (int)threadIdx.x * run), w1 = min(W, w0 + run);
    int n = 0;
    for (int w = w0; w < w1; w++) n += __popc(*(volatile unsigned*)(map + w));
    int s = n;
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
        const int y = __shfl_up_sync(kAll, s, d);
        if (lane >= d) s += y;
    }
    if (lane == 31) warps[warp] = s;
    __syncthreads();
    int at = s - n;
    for (int w = 0; w < warp; w++) at += warps[w];
    for (int w = w0; w < w1; w++) {
        pre[w] = at;
        unsigned bits = *(volatile unsigned*)(map + w);
        while (bits) {
            const int row = w * 32 + __ffs(bits) - 1;
            a.cell_e[c0 + at++] = row * a.g.jp + j;
            bits &= bits - 1;
        }
    }
    for (int c = threadIdx.x; c < nc; c += NT) owner[c] = 0x7fffffff;
    if (threadIdx.x == 0) placed = 0;
    __syncthreads();
    // each marker's nine places
    int* place = a.place + (size_t)9 * p0;
    for (int p = threadIdx.x; p < m; p += NT) {
        int row[9];
        stencil_rows(a.markers[a.by_plane[p0 + p]], a.g, row);
#pragma unroll
        for (int c = 0; c < 9; c++) {
            const int w = row[c] >> 5;
            place[9 * p + c] = *(volatile int*)(pre + w) + __popc(*(volatile unsigned*)(map + w) & ((1u << (row[c] & 31)) - 1u));
        }
    }
    __syncthreads();
    int level = 0;
    if (m <= kHeld * NT) {
        // every thread holds its markers' places (kHeld sets of nine)
        int pl[kHeld][9], q[kHeld];
        bool left[kHeld];
#pragma unroll
        for (int u = 0; u < kHeld; u++) {
            const int p = u * NT + (int)threadIdx.x;
            left[u] = p < m;
            q[u] = left[u] ? a.by_plane[p0 + p] : 0;
#pragma unroll
            for (int c = 0; c < 9; c++) pl[u][c] = left[u] ? place[9 * p + c] : 0;
        }
        int done = 0;
        for (; level < kMaxRounds; level++) {
#pragma unroll
            for (int u = 0; u < kHeld; u++)
                if (left[u])
#pragma unroll
                    for (int c = 0; c < 9; c++) atomicMin(owner + pl[u][c], u * NT + (int)threadIdx.x);
            __syncthreads();
            unsigned vote[kHeld];
            bool ready[kHeld];
#pragma unroll
            for (int u = 0; u < kHeld; u++) {
                ready[u] = left[u];
                if (left[u])
#pragma unroll
                    for (int c = 0; c < 9; c++) ready[u] = ready[u] && *(volatile int*)(owner + pl[u][c]) == u * NT + (int)threadIdx.x;
                vote[u] = __ballot_sync(kAll, ready[u]);
                if (lane == 0) counts[u][warp] = __popc(vote[u]);
            }
            __syncthreads();
#pragma unroll
            for (int u = 0; u < kHeld; u++) {
                // the counts of the warps before this one, and of all
                int x = lane < NT / 32 ? counts[u][lane] : 0;
                const int before = __reduce_add_sync(kAll, lane < warp ? x : 0), all = __reduce_add_sync(kAll, x);
                if (ready[u]) {
                    const int slot = p0 + done + before + __popc(vote[u] & ((1u << lane) - 1u));
                    a.sched[slot] = q[u];
                    float* prep = a.prep + (size_t)slot * PF_STRIDE + PF_CELL;
#pragma unroll
                    for (int c = 0; c < 9; c++) {
                        prep[c] = __int_as_float(pl[u][c]);
                        owner[pl[u][c]] = 0x7fffffff;   // (this round's cells of one marker are no other's)
                    }
                    left[u] = false;
                }
                done += all;
            }
            if (threadIdx.x == 0) a.level_end[p0 + level] = p0 + done;
            // (cells of no placed marker hold the lowest of those that wait, and keep it)
            __syncthreads();
            if (done == m) break;
        }
        if (threadIdx.x == 0) {
            a.levels[j] = level + 1;
            if (level == kMaxRounds) atomicExch(a.info + 1, 1);
        }
        return;
    }
    for (; level < kMaxRounds; level++) {
        for (int p = threadIdx.x; p < m; p += NT) {
            if (place[9 * p] < 0) continue;
#pragma unroll
            for (int c = 0; c < 9; c++) atomicMin(owner + place[9 * p + c], p);
        }
        __syncthreads();
        for (int b = 0; b < m; b += NT) {
            const int p = b + (int)threadIdx.x;
            bool ready = p < m && place[9 * p] >= 0;
            int pl[9];
            if (ready) {
#pragma unroll
                for (int c = 0; c < 9; c++) {
                    pl[c] = place[9 * p + c];
                    ready = ready && *(volatile int*)(owner + pl[c]) == p;
                }
            }
            const unsigned vote = __ballot_sync(kAll, ready);
            if (lane == 0) warps[warp] = __popc(vote);
            __syncthreads();
            int before = placed, all = 0;
#pragma unroll
            for (int w = 0; w < NT / 32; w++) {
                if (w < warp) before += warps[w];
                all += warps[w];
            }
            if (ready) {
                const int slot = p0 + before + __popc(vote & ((1u << lane) - 1u));
                a.sched[slot] = a.by_plane[p0 + p];
                float* prep = a.prep + (size_t)slot * PF_STRIDE + PF_CELL;
#pragma unroll
                for (int c = 0; c < 9; c++) prep[c] = __int_as_float(pl[c]);
                place[9 * p] = -1;   // placed (the thread's own marker in every round)
            }
            __syncthreads();
            if (threadIdx.x == 0) placed += all;
            __syncthreads();
        }
        if (threadIdx.x == 0) a.level_end[p0 + level] = p0 + placed;
        for (int c = threadIdx.x; c < nc; c += NT) owner[c] = 0x7fffffff;
        __syncthreads();
        if (placed == m) break;
    }
    if (threadIdx.x == 0) {
        a.levels[j] = level + 1;
        if (level == kMaxRounds) atomicExch(a.info + 1, 1);
    }
}

// Levels before each plane; the (empty) second segment starts after all of them.
__global__ void __launch_bounds__(1024) k_sched_finish(SchedArgs a) {
    for (int j = threadIdx.x; j < a.g.ny; j += 1024) a.plane_lv0[j] = a.levels[j];
    __syncthreads();
    const int total = block_scan(a.plane_lv0, a.g.ny);
    for (int j = threadIdx.x; j <= a.g.ny; j += 1024) a.plane_lv1[j] = total;
    if (threadIdx.x == 0) {
        a.info[2] = total;
        if (a.info[1] == 0) a.level_ptr[total] = a.n0;
    }
}

__global__ void __launch_bounds__(128) k_sched_level_ptr(SchedArgs a) {
    if (a.info[1]) return;   // given up: the levels are not whole
    const int j = (int)blockIdx.x, p0 = a.plane_slot[j], lv = a.plane_lv0[j];
    for (int r = threadIdx.x; r < a.levels[j]; r += 128) a.level_ptr[lv + r] = r == 0 ? p0 : a.level_end[p0 + r - 1];
}

__global__ void __launch_bounds__(256) k_static_flags(Dims g, const int* __restrict__ cell_e, int n, uint32_t* __restrict__ mask) {
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (t >= n) return;
    const int e = cell_e[t], row = e / g.jp, j = e - row * g.jp;
    atomicOr(mask + (long long)row * g.jw + (j >> 5), 1u << (j & 31));
}

// ---------------------------------------------------------------------------
constexpr size_t kMapSmem = 160 * 1024;   // shared memory the two maps may take

size_t sched_hist_ints(const Dims& g, long long n) { return (size_t)((n + chunk_of(n) - 1) / chunk_of(n)) * (size_t)g.ny; }
size_t sched_map_words(const Dims& g) {
    const size_t W = (size_t)((g.rows() + 31) / 32);
    return W * 8 <= kMapSmem ? 0 : 2 * W * (size_t)g.ny;
}

cudaError_t launch_sched_cells(const SchedArgs& a, cudaStream_t st) {
    const int per = chunk_of(a.n), nchunk = (int)((a.n + (long long)per - 1) / per);
    if (nchunk > 0) k_sched_count<<<(nchunk + 3) / 4, 128, 0, st>>>(a, nchunk, per);
    k_sched_offsets<<<(a.g.ny + 3) / 4, 128, 0, st>>>(a, nchunk);
    k_sched_scan<<<1, 1024, 0, st>>>(a);
    if (nchunk > 0) k_sched_scatter<<<(nchunk + 3) / 4, 128, 0, st>>>(a, nchunk, per);
    const size_t smem = a.maps ? 0 : (size_t)((a.g.rows() + 31) / 32) * 4;
    cudaError_t e = raise_smem_limit((const void*)k_sched_cells, smem);
    if (e != cudaSuccess) return e;
    k_sched_cells<<<a.g.ny, 256, smem, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_sched_levels(const SchedArgs& a, int max_cells, int ncell, cudaStream_t st) {
    const size_t maps = a.maps ? 0 : (size_t)((a.g.rows() + 31) / 32) * 8;
    // owner arrays in shared memory for the planes whose cells fit in what is left
    const int cap = (int)std::min<size_t>((size_t)max_cells, (220 * 1024 - maps) / 4);
    const size_t smem = maps + (size_t)cap * 4;
    cudaError_t e = raise_smem_limit((const void*)k_sched_levels<512>, smem);
    if (e != cudaSuccess) return e;
    k_sched_levels<512><<<a.g.ny, 512, smem, st>>>(a, cap);
    k_sched_finish<<<1, 1024, 0, st>>>(a);
    k_sched_level_ptr<<<a.g.ny, 128, 0, st>>>(a);
    if (ncell > 0) k_static_flags<<<(ncell + 255) / 256, 256, 0, st>>>(a.g, a.cell_e, ncell, a.mask_static);
    return cudaGetLastError();
}

}  // namespace tdlb
