// Internal interface between the host runtime (tdlb_capi.cu) and the kernels.
#pragma once
#include <atomic>
#include "tdlb_common.cuh"

namespace tdlb {

// Which cells a step launch takes (step_kernels.cuh). Cells are told apart by
// flag words, the 32 cells of a row whose touched flags share a word: part 1
// takes the words whose `skip` byte is zero, part 2 the words of a list (NULL:
// the first `count`), without the cells whose bit is set in `except` (NULL: all
// of them). Part 0 takes every cell. l2_ahead > 0 turns on the L2 prefetch of
// parts 0 and 1, that many CTAs ahead of the walk.
struct StepPart {
    const uint8_t* skip;
    const int* words;
    int count;
    const uint32_t* except;
    int l2_ahead;
};

// Part 2: 32 / V lanes of a 128-thread block share a word of the list. Words are
// counted, not threads: a lattice of a few cells along y has a word per row, up
// to 2^30 of them, and 32 threads a word pass 2^32.
__host__ __device__ inline unsigned listed_word(unsigned block, unsigned thread, unsigned V) {
    return block * (4u * V) + thread * V / 32u;
}
inline unsigned listed_blocks(long long words, unsigned V) { return (unsigned)((words + 4u * V - 1) / (4u * V)); }

// One wave of resident 128-thread CTAs of kernel K on the current device (the
// occupancy its register count allows, times the SMs): the L2 prefetch
// distance of a full launch. Queried once per kernel; 0 (prefetch off) if the
// query fails.
template <auto K>
int wave_ctas() {
    static std::atomic<int> n{0};
    int v = n.load(std::memory_order_relaxed);
    if (v == 0) {
        int dev = 0, sms = 0, per = 0;
        if (cudaGetDevice(&dev) == cudaSuccess &&
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, K, 128, 0) == cudaSuccess && per > 0 && sms > 0) {
            v = per * sms;
            n.store(v, std::memory_order_relaxed);
        }
    }
    return v;
}

// A launch whose blocks are set up while the stream's previous launch drains.
// Every thread of such a kernel begins with after_previous(), which returns
// once that launch has ended and its writes are visible: the order on the
// stream is that of an ordinary launch. In a kernel with read-only loads (const
// __restrict__ or __ldg) the index that addresses them goes through it, so that
// none of them can be moved ahead of it (k_ibm_gather has none; there the index
// through it cost registers: 192^3 BF16 30.5 -> 34.9 us).
// The step, gather, spread, load and rotation of a small tank are a chain of
// launches of 2 to 25 us with 1.5 to 3 us between them. B200, runs of 60 steps
// with forcing, load and rotation, ordinary launches -> these: 24^3 2.86 ->
// 2.14 ms, 101x83x97 with uploaded blades 5.44 -> 5.03, 160^3 FP16 Simple 9.55
// -> 9.12, 192^3 BF16 Esotwist 13.06 -> 12.97, 400^3 FP16 Esotwist 64.4 -> 64.6
// (equal). A captured stream gets ordinary launches.
template <typename... P, typename... A>
cudaError_t launch_chained(void (*kernel)(P...), unsigned grid, int block, size_t smem, cudaStream_t st, A... args) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &capture) != cudaSuccess) return cudaGetLastError();
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = capture == cudaStreamCaptureStatusNone ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
    return cudaGetLastError();
}
__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" : : : "memory"); }
template <typename T>
__device__ __forceinline__ void after_previous(T& index) {
    static_assert(sizeof(T) == 4, "a 32-bit index");
    asm volatile("griddepcontrol.wait;" : "+r"(index) : : "memory");
}

// Arguments of one fused step launch.
struct StepArgs {
    Planes A;               // Simple: source buffer; Esotwist: the single buffer
    Planes B;               // Simple: destination buffer (unused for Esotwist)
    float* Nu;
    const float4* F;        // force, one float4 (Fx, Fy, Fz, unused) per element
    const uint32_t* mask;   // IBM-touched flags of the forcing pass this step uses
    Dims g;
    CollideParams p;
    int les;                // Smagorinsky LES on/off (FlowParams::useLES)
    int from_moments;       // state holds moments (after initialise / checkpoint load)
    int collide;            // 0: transport only (identity collision; known-answer tests)
    int even;               // Esotwist parity (evenStep)
    int vec;                // cells per thread: 1, 2 or 4 (float, float2, float4 traffic)
    int l2_prefetch;        // full launches of the population form: L2 prefetch one wave ahead
    int storage;            // StorageKind of the population planes
    int part;               // 0: every cell; 1: outer words; 2: inner words (populations; FP32: vec == 1)
    StepPart zone;          // the words of part 1 or 2
    ResidualBox rr;         // 16-bit storage: residuals of the locations read ...
    ResidualBox rw;         // ... and written (Simple: of buffer A and B; Esotwist: the same box)
    const int* box_cells;   // elements of the cells the box launch steps
    int n_box;
};

// The StepPart a launch of kernel K takes: a.zone, with, for a launch over the
// whole lattice of the population form (FULL) and a.l2_prefetch on, the L2
// prefetch distance of one wave of K's resident CTAs.
template <auto K, bool FULL>
StepPart launch_walk(const StepArgs& a) {
    StepPart w = a.zone;
    w.l2_ahead = FULL && a.part != 2 && a.l2_prefetch ? wave_ctas<K>() : 0;
    return w;
}

cudaError_t launch_step_simple(const StepArgs& a, cudaStream_t st);
cudaError_t launch_step_esotwist(const StepArgs& a, cudaStream_t st);
cudaError_t launch_step_simple_h16(const StepArgs& a, cudaStream_t st);
cudaError_t launch_step_esotwist_h16(const StepArgs& a, cudaStream_t st);
// The box cells of a step with a residual box (the other launches leave them out).
cudaError_t launch_box(const StepArgs& a, bool simple, cudaStream_t st);

// ---- the zone of a split step (zone.cu) ----
// core: a bit for every cell in a stencil of the resident markers at any
// impeller angle: the static flags, and per plane j the annulus
// [ring[j].x, ring[j].y] about (ci, ck) (none where y < 0).
cudaError_t launch_zone_core(const Dims& g, const uint32_t* mask_static, const double2* ring, double ci, double ck,
                             uint32_t* core, cudaStream_t st);
// skip: a byte per word, 1 where the word holds a core cell or (neighbours) a
// periodic neighbour of one.
cudaError_t launch_zone_words(const Dims& g, const uint32_t* core, int neighbours, uint8_t* skip, cudaStream_t st);
// Box cells: their bits in `except` (zeroed by the caller), their words in skip;
// either may be NULL.
cudaError_t launch_zone_box(const Dims& g, const int* cells, int n, uint32_t* except, uint8_t* skip, cudaStream_t st);
cudaError_t launch_fill_uniform_moments(Planes Q, const Dims& g, float rho, cudaStream_t st);

// ---- immersed boundary ----

// Marker record, identical in layout to tdlb_marker (include/tdlb_b200.h).
struct Marker {
    long long i, j, k;
    float iCartFraction, kCartFraction, uDelta, vDelta, wDelta, pad;
};
static_assert(sizeof(Marker) == 48, "Marker layout");

// Blade (second-segment) scratch written by k_ibm_gather, read by the
// spread walk; field-major over the segment's slots.
enum TailField {
    TF_W = 0,               // 9 stencil weights, (k1, i1) order
    TF_RHO = 9,             // 9 densities
    TF_MX = 18, TF_MY = 27, TF_MZ = 36,   // 9 momenta each
    TF_U = 45, TF_V = 46, TF_WV = 47,     // marker velocity
    TF_CELL = 48,           // 9 packed (i << 16 | k) cells (int32 bit patterns)
    TF_COUNT = 57
};

// First-segment (static markers) data prepared once per upload, per slot
// p < n0: 9 weights, 9 plane-local cell indices, the marker velocity.
enum PrepField {
    PF_W = 0,
    PF_CELL = 9,            // int32 bit patterns
    PF_U = 18, PF_V = 19, PF_WV = 20,
    PF_STRIDE = 24          // floats per marker: marker-major rows of 96 bytes (six float4 loads)
};

struct IbmArgs {
    const Marker* markers;      // device copy of the marker list (list order)
    const int* sched;           // execution order: marker index per slot
    const int* level_ptr;       // [nlevels+1] slot offsets of each level
    const int* plane_lv0;       // [ny+1] levels of each j-plane, first segment
    const int* plane_lv1;       // [ny+1] levels of each j-plane, second segment (walked after the first)
    int n;                      // number of markers
    int n0;                     // markers (slots) of the first segment
    // first segment: unique stencil cells, sorted by (j, i, k)
    const int* cell_e;          // [C0] element index of each cell
    const int* plane_cell;      // [ny+1] cell range of each plane
    int ncell;                  // C0
    int max_cells, max_big;     // most cells of an ordinary plane, of a big plane
    const float* prep;          // PF_STRIDE * n0: one row per first-segment slot
    float* cell_m;              // C0 float4: rho, jx, jy, jz of each cell this pass
    float* cell_F;              // 3 * C0: F of each cell at the start of this pass
    float* tail;                // TF_COUNT * ntail_cap
    long long tail_cap;
    float* sums;                // 3 * n: each slot's spread sums (for the impeller load)
    int smem_cells;             // F tile capacity of the small-plane launch
    const int* plane_list;      // [ny] small planes first, then the big ones
    int n_small, n_big;         // planes in each launch
    const int* blade_planes;    // the planes with blade levels (the blade launch)
    int n_blade, blade_words;   // their count; shared-memory floats of the blade launch
    int blade_max, pad0;        // most blade markers of a plane
    int big_tile_cells;         // F tile capacity of the big-plane launch
    cudaStream_t side;          // stream of the big-plane launch
    cudaEvent_t ev_fork, ev_join;
    Planes A;                   // current state
    int state_mode;             // 0 Simple pops, 1 moments, 2 Esotwist pops, 3 Esotwist moments
    int even;                   // Esotwist parity of the state's read map
    float4* F4;                 // force, one float4 (Fx, Fy, Fz, unused) per element
    const uint32_t* mask_old;   // touched flags of the previous forcing pass
    uint32_t* mask_new;         // touched flags of this pass (fully written)
    const uint32_t* mask_static;   // touched flags of the first segment (every pass)
    size_t mask_bytes;
    Dims g;
    float alpha, beta;
    int storage;                // StorageKind of the state planes
    CollideParams p;            // rest offsets of the 16-bit storage
    ResidualBox rbox;           // residuals of the state's locations (16-bit storage; off: res == NULL)
};

cudaError_t launch_ibm(const IbmArgs& a, cudaStream_t st);

// ---- the marker scheduler on the device (schedule.cu) ----
struct SchedArgs {
    const Marker* markers;      // the list
    int n, n0;                  // its length, the first segment's
    Dims g;
    // scratch
    int* info;                  // [3] first marker out of range (starts at n), given up (starts at 0), levels
    int* hist;                  // [sched_hist_ints] zero
    int* by_plane;              // [n0]
    unsigned* maps;             // [sched_map_words], NULL when that is 0
    int* place;                 // [9 n0]
    int* owner;                 // [cells]
    int* level_end;             // [n0]
    int* levels;                // [ny]
    // results of launch_sched_cells
    int* plane_slot;            // [ny+1] slots of each plane
    int* plane_count;           // [ny] unique stencil cells of each plane
    // inputs and results of launch_sched_levels
    const int* plane_cell;      // [ny+1] running sum of plane_count
    int* cell_e;                // [cells]
    int* sched;                 // [n0]
    float* prep;                // [PF_STRIDE n0]: the places (PF_CELL)
    int* level_ptr;             // [levels + 1]
    int* plane_lv0;             // [ny+1]
    int* plane_lv1;             // [ny+1]: an empty second segment
    uint32_t* mask_static;      // zero; touched flags of the cells
};
size_t sched_hist_ints(const Dims& g, long long n);
size_t sched_map_words(const Dims& g);
// The list checked and sorted by plane, the planes' cells counted.
cudaError_t launch_sched_cells(const SchedArgs& a, cudaStream_t st);
// Cells, levels and order; max_cells: the most of a plane, ncell: of all.
cudaError_t launch_sched_levels(const SchedArgs& a, int max_cells, int ncell, cudaStream_t st);
// Raise a kernel's dynamic shared-memory limit on the current device (it only grows).
cudaError_t raise_smem_limit(const void* fn, size_t bytes);

// Immersed-boundary passes of many lattices in one set of launches: device
// IbmArgs per lattice and work lists. gather: GatherItem's; small / big:
// (lattice, j-plane), 128 / 512 threads.
enum GatherKind { GATHER_CELLS = 0, GATHER_TAIL = 1, GATHER_FLAGS = 2 };
// A block's work of the gather: the kind and the lattice (x); the tile of 32
// planes and kCellPlaces places (CELLS), or a number of 256 (blade marker, cell)
// pairs or of kMaskCopyWords touched-flag words (y). The place's upper bits stand
// beside the lattice, so that a plane may have any number of cells (all of it in y
// with the kind ran out at 2^22). The shift that takes the place out of y is a
// signed one: where the compiler can tell that the place is not negative (unsigned,
// or a word of its own) the tile's code is slower, 64 FP16 tanks 1.477 -> 1.498 ms
// a step.
constexpr int kCellPlaces = 8;
struct GatherItem {
    int tank, kind, y, upper;
    __host__ __device__ static int2 cells(int tank, int j0, int p0) {
        const int place = p0 / kCellPlaces;
        return make_int2(place >> 21 << 24 | tank << 2 | GATHER_CELLS, (place & 0x1fffff) << 10 | j0 / 32);
    }
    __host__ __device__ static int2 other(int tank, int kind, int number) { return make_int2(tank << 2 | kind, number); }
    __host__ __device__ static GatherItem of(int2 w) { return GatherItem{(w.x >> 2) & 0x3fffff, w.x & 3, w.y, w.x >> 24}; }
    __host__ __device__ int j0() const { return (y & 0x3ff) * 32; }
    __host__ __device__ int p0() const { return ((y >> 10) + (upper << 21)) * kCellPlaces; }
};
struct IbmBatch {
    const IbmArgs* args;
    const int2* gather; int n_gather;
    const int2* small; int n_small;
    const int2* big; int n_big;
    int small_tile, big_tile;   // dynamic F tiles (cells) of the two spread launches
    int storage;
};
constexpr int kMaskCopyWords = 8192;
cudaError_t launch_ibm_batch(const IbmBatch& b, cudaStream_t st, cudaStream_t side, cudaEvent_t fork, cudaEvent_t join);
cudaError_t ibm_batch_prepare_smem(int small_cells, int big_cells);
// Per-upload preparation of the first segment (weights, velocities).
cudaError_t launch_ibm_prepare(const IbmArgs& a, float* prep, cudaStream_t st);
// Opt the spread kernels in to the dynamic shared memory of the ordinary
// planes' launch (tiles of `small_cells` cells) and of the big planes'
// launch (`big_bytes`).
cudaError_t ibm_prepare_smem(int small_cells, size_t big_bytes);
// Shared memory of the big planes' launch for a tile of `big_cells` cells.
size_t big_bulk_bytes(int big_cells);
// Shared-memory floats of the blade launch for a plane of nb blade markers,
// and the opt-in to that many.
int blade_table_words(int nb);
cudaError_t ibm_prepare_blades(int words);
// FP64 force and torque of the impeller's slots of the last forcing pass:
// out[0..2] = -beta * sum of spread sums, out[3] = torque about the tank axis
// (ci, ck), out[4] = number of markers summed. `partial` holds kLoadBlocks * 5
// doubles, `counter` is zero between launches.
constexpr int kLoadBlocks = 128;
cudaError_t launch_marker_load(const IbmArgs& a, const int* slots, int n, double ci, double ck, double* partial,
                               unsigned* counter, double* out, cudaStream_t st);
// Slots of the markers with list index >= begin, ascending: slots NULL: their
// number in each group of 256 slots to `offset`; else to slots, from each
// group's offset.
cudaError_t launch_impeller_slots(const int* sched, int n, int begin, int* offset, int* slots, cudaStream_t st);
// FP64 mass/momentum reduction: out[0] = sum rho, out[1..3] = sum (j + F/2).
// `partial` holds kReduceBlocks * 4 doubles.
constexpr int kReduceBlocks = 592;
cudaError_t launch_reduce_fp64(const IbmArgs& a, const uint32_t* mask, double* partial, double* out, cudaStream_t st);
// Rest state at density rho for the 16-bit storage.
cudaError_t launch_fill_rest(Planes Q, long long plane, float rho, float rho0, int storage, const CollideParams& p,
                             cudaStream_t st);
// The parts of a blade upload from `stage`, one after another: n markers, their
// order, nlev level offsets, nplane plane levels.
cudaError_t launch_place_blades(const int* stage, Marker* markers, int n, int* order, int* level_ptr, int nlev, int* plane_lv,
                                int nplane, cudaStream_t st);
// Recompute n rotating markers (offsets xz[2n]) for cos/sin (ca, sa).
cudaError_t launch_rotate_markers(const double* xz, Marker* out, int n, double ca, double sa, double omega, double ci,
                                  double ck, int nx, int nz, cudaStream_t st);

}  // namespace tdlb
