// The handle behind tdlb_handle (include/tdlb_b200.h): one lattice on one
// GPU with its device buffers, resident markers and state bookkeeping.
// Shared by the C-ABI translation units.
#pragma once

#include <string>
#include <vector>

#include "tdlb_b200.h"
#include "tdlb_kernels.cuh"
#include "tdlb_runtime.hpp"

using tdlb::Dims;
using tdlb::Planes;

struct tdlb_lattice {
    tdlb_config cfg{};
    Dims g{};
    int device = 0;
    cudaStream_t stream = nullptr;       // all of the handle's work is queued here
    cudaStream_t own_stream = nullptr;   // set when `stream` is borrowed from a batch
    tdlb::CollideParams cp{};

    char* block = nullptr;       // one allocation: the five arrays below (tdlb_rt::LatticeBlock)
    float* bufA = nullptr;       // 18 planes
    float* bufB = nullptr;       // 18 planes (Simple only)
    float* Nu = nullptr;
    float* F = nullptr;          // a float4 (Fx, Fy, Fz, unused) per element
    uint32_t* mask = nullptr;    // 2 x (rows * jw) words
    long long mask_words = 0;

    // state
    int cur = 0;                 // Simple: which buffer holds the state (0 A, 1 B)
    bool holds_moments = true;   // state is in moment form (after initialise)
    bool even = true;            // Esotwist parity (ComputeUnit.hpp:116)
    int pass = 0;                // forcing passes so far; mask[pass & 1] is current
    int vec = 4;                 // cells per thread of the step kernels (set per scheme in build())
    int l2_prefetch = 1;         // full step launches prefetch one wave ahead into L2 (tdlb_set_l2_prefetch)
    bool initialised = false;

    // markers: the resident list and its two-segment schedule
    tdlb::Marker* d_markers = nullptr;
    int* d_sched = nullptr;
    int* d_level_ptr = nullptr;
    int* d_plane_lv0 = nullptr;
    int* d_plane_lv1 = nullptr;
    // first-segment cell lists and per-pass IBM buffers (grown on demand)
    std::vector<int> plane_cell;  // [ny+1] cell range of each plane (empty: none yet)
    int ncell = 0;                // unique stencil cells
    int n_level0 = 0;             // levels of the first segment
    long long cell_cap = 0, prep_cap = 0;
    tdlb::Marker* d_markers_in = nullptr;   // the next list, until it has been checked
    void* d_sched_tmp = nullptr;  // scratch of the scheduler
    size_t sched_tmp_bytes = 0;
    int* d_cell_e = nullptr;
    int max_cells = 0, max_big = 0;   // most cells of an ordinary plane, of a big plane
    int* d_plane_cell = nullptr;
    float* d_prep = nullptr;      // PF_STRIDE * n0
    float* d_cell_m = nullptr;    // 4 * C0 (float4 per cell)
    float* d_cell_F = nullptr;    // 3 * C0
    float* d_tail = nullptr;      // TF_COUNT * tail_cap
    long long tail_cap = 0;
    float* d_sums = nullptr;      // 3 * marker_cap
    int smem_cells = 0;
    int* d_plane_list = nullptr;  // small planes, then big planes
    std::vector<int> h_plane_list;   // host copy of d_plane_list
    unsigned marker_gen = 0;      // bumped by every marker upload
    int n_small = 0, n_big = 0, big_tile_cells = 0;
    // the planes with blade levels, walked by their own launch
    std::vector<int> h_blade_planes;
    int* d_blade_planes = nullptr;
    int n_blade = 0, blade_words = 0, blade_max = 0;
    cudaStream_t side = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    uint32_t* d_mask_static = nullptr;   // first segment's touched cells
    uint32_t* d_exclude = nullptr;       // excluded output points (1 bit per cell), when set
    std::vector<uint32_t> h_exclude;
    double* d_red = nullptr;             // FP64 reduction partials + result
    long long marker_cap = 0, marker_in_cap = 0;   // of d_markers, d_markers_in
    long long slot_cap = 0;                         // of d_sched, d_sums
    long long level_cap = 0;
    int n_markers = 0;      // list length
    int n0 = 0;             // markers of the first segment (the rest rotate)
    std::vector<tdlb_marker> h_blades;    // host copy of the second segment
    tdlb::MarkerSchedule seg1;
    bool markers_set = false;
    float last_beta = 0.f;        // beta of the last forcing pass (for the load)
    // resident impeller: markers [n0, n_markers) are blades
    char* imp_block = nullptr;    // one allocation: the impeller's arrays (d_rot_xz, d_load, d_imp_slots, d_blade_stage)
    size_t imp_block_cap = 0;
    double* d_rot_xz = nullptr;   // their impeller-frame offsets (device rotation)
    bool rot_device = false;
    double rot_ci = 0, rot_ck = 0;
    int impeller_begin = -1;      // first marker of the impeller (-1: none)
    tdlb_rushton rspec{};         // the attached impeller's spec
    double angle = 0.0;           // impeller angle of the last rotation
    unsigned long long rstep = 1; // main-loop step the angle belongs to (main.cpp:336 starts at 1)
    double* d_load = nullptr;     // kLoadBlocks*5 partials + 5 results + a counter
    int* d_imp_slots = nullptr;   // the impeller's slots, ascending
    int n_imp = 0;
    // pinned staging of the per-step blade upload (markers and their
    // schedule), two buffers used in turn; each buffer's event marks the end
    // of the copies that read it
    struct PinStage {
        char* p = nullptr;
        size_t cap = 0;
        cudaEvent_t ev = nullptr;
    } pin[2];
    int pin_cur = 0;
    char* d_blade_stage = nullptr;   // the upload on the device, before its parts are placed
    std::vector<double> h_rot_xz; // host copy of d_rot_xz
    std::vector<int> h_rot_j;     // and the planes of those blades

    // Split steps: the outer words of a step run on `bulk`, beside the previous
    // forcing pass and the inner words on `stream`, which then waits for them:
    // work queued on `stream` after a step sees all of it.
    cudaStream_t bulk = nullptr;
    cudaEvent_t ev_outer = nullptr, ev_inner = nullptr, ev_fence = nullptr;
    int overlap = -1;             // split steps: 0 off, 1 when the zone is small, 2 always (tdlb_set_overlap);
                                  // -1: as 1, for lattices large enough
    bool bulk_ok = false;         // nothing but step-loop work queued since ev_inner: the next outer
                                  // launch waits for that event alone
    bool stream_taken = false;    // the caller has the stream (tdlb_get_stream) and may queue work there that the
                                  // next step has to follow: no step splits unasked from then on
    bool resident = false;        // markers kept for many passes (set/attach), so a zone pays
    // the zone (zone.cu), for marker_gen zone_gen and box_gen zone_box_gen; its
    // arrays are one allocation, made where the markers are set (tdlb_rt::
    // reserve_zone): a step allocates nothing, and without them does not split
    unsigned zone_gen = ~0u, zone_box_gen = ~0u;
    bool zone_ok = false;         // every stencil cell of the current markers lies in it
    bool zone_small = false;      // it holds at most 60 % of the cells
    char* zone_block = nullptr;
    uint32_t* d_zone_core = nullptr;     // 1 bit per cell: the stencil cells
    int* d_zone_words = nullptr;         // the zone's words, ascending
    double2* d_zone_ring = nullptr;      // per plane: radii of the blades' annulus
    uint8_t* d_zone_skip = nullptr;      // 1 byte per flag word: in the zone
    int n_zone = 0, n_outer = 0;         // words inside, outside
    int list_passes = 0;          // forcing passes (or batch runs) of the resident list so far
    // the last forcing pass, which F and the current flags are of
    bool forced = false;          // there was one since F was last zero everywhere
    unsigned force_gen = ~0u;     // marker_gen of its list (~0: not known)
    bool force_blades_in = false; // its blades lay inside the zone of that list
    std::vector<uint8_t> h_zone_skip;
    std::vector<uint32_t> h_zone_core;   // filled when host blades are checked against it
    // 16-bit storage: the residual box (tdlb::ResidualBox) and its residuals,
    // one set per population buffer (Simple: A and B; Esotwist: one)
    tdlb::ResidualBox rbox_geom{};        // geometry only (res unused)
    float* d_res[2] = {nullptr, nullptr};
    bool rbox_auto = true;                // set from the impeller by tdlb_attach_rushton
    unsigned box_gen = 0;                 // bumped by every change of the box
    // the cells that the box launch of a step takes: their elements, ascending,
    // and a bit for each (the other launches leave them out)
    int* d_box_list = nullptr;
    int n_box = 0;
    uint32_t* d_box_except = nullptr;
    // device scratch of the read-back (a slab of output) and the plane dumps
    void* d_scratch = nullptr;
    size_t scratch_bytes = 0;
    // step-kernel timing (tdlb_set_kernel_timing): start/stop event pairs
    bool timing = false;
    std::vector<cudaEvent_t> tev;
    long long launches = 0;       // kernels queued by the step loop (tdlb_kernel_launches)

    std::string err = "no error";

    size_t esz() const { return cfg.storage == TDLB_STORAGE_FP32 ? 4 : 2; }   // bytes per population
    Planes planes(float* base) const {
        Planes p;
        for (int d = 0; d < tdlb::NQ; d++)
            p.p[d] = reinterpret_cast<float*>(reinterpret_cast<char*>(base) + (size_t)d * (size_t)g.plane * esz());
        return p;
    }
    // FP32 planes of a moment buffer (always FP32)
    Planes planes32(float* base) const {
        Planes p;
        for (int d = 0; d < tdlb::NQ; d++) p.p[d] = base + (size_t)d * (size_t)g.plane;
        return p;
    }
    // residual box of population buffer `buf` (0: bufA, 1: bufB); off when
    // no box is set
    tdlb::ResidualBox rbox(int buf) const {
        tdlb::ResidualBox b = rbox_geom;
        b.res = d_res[buf];
        return b;
    }
    int state_index() const { return cfg.streaming == TDLB_STREAMING_SIMPLE && cur == 1 ? 1 : 0; }
    float* state_buf() const { return cfg.streaming == TDLB_STREAMING_SIMPLE && cur == 1 ? bufB : bufA; }
    float* other_buf() const { return cur == 1 ? bufA : bufB; }
    uint32_t* mask_cur() const { return mask + (size_t)(pass & 1) * mask_words; }
    uint32_t* mask_next() const { return mask + (size_t)((pass + 1) & 1) * mask_words; }
    int state_mode() const {
        if (cfg.streaming == TDLB_STREAMING_SIMPLE) return holds_moments ? 1 : 0;
        return holds_moments ? 3 : 2;
    }
};


// Runtime helpers shared by the C-ABI translation units (tdlb_capi.cu).
namespace tdlb_rt {
// Default cells per thread of a lattice's step kernel. Measured on B200 at
// 400^3 with the L2 prefetch on (step kernel alone, one, two, four cells): FP32
// Simple 1.462, 1.475, 1.575 ms, Esotwist 1.483, 1.522, 1.582; 16-bit storage with
// packed FP32x2 arithmetic, Simple 1.176, 1.072, 0.905, Esotwist 1.335, 1.081,
// 1.143.
inline int default_cells_per_thread(const tdlb_config& c) {
    if (c.storage == TDLB_STORAGE_FP32) return 1;
    return c.streaming == TDLB_STREAMING_SIMPLE ? 4 : 2;
}
// The lattice's arrays in one device allocation, each on a 256-byte boundary:
// an allocation above a megabyte takes about 0.7 ms and its free as long, four or
// five times over for every tank that a server builds.
struct LatticeBlock {
    size_t a, b, nu, f, mask, bytes;   // offsets; b == a without a second buffer
    void place(tdlb_lattice* h, char* base) const {
        h->bufA = (float*)(base + a);
        h->bufB = b == a ? nullptr : (float*)(base + b);
        h->Nu = (float*)(base + nu);
        h->F = (float*)(base + f);
        h->mask = (uint32_t*)(base + mask);
    }
    void place(tdlb_lattice* h) const { place(h, h->block); }
};
inline LatticeBlock lattice_block(const Dims& g, long long mask_words, size_t esz, bool simple) {
    auto up = [](size_t n) { return (n + 255) / 256 * 256; };
    const size_t pop = up((size_t)tdlb::NQ * g.plane * esz), plane = up((size_t)g.plane * sizeof(float));
    LatticeBlock l{};
    l.b = simple ? pop : 0;
    l.nu = l.b + pop;
    l.f = l.nu + plane;
    l.mask = l.f + 4 * plane;          // F: one float4 per element
    l.bytes = l.mask + up((size_t)2 * mask_words * sizeof(uint32_t));
    return l;
}
// The message of a CUDA call that failed. The runtime also keeps the error for
// cudaGetLastError, where the next call's launch check would find it: an
// allocation that failed is told of once.
inline std::string error_text(const char* call, cudaError_t e) {
    cudaGetLastError();
    return std::string(call) + ": " + cudaGetErrorString(e);
}
tdlb::StepArgs step_args(tdlb_lattice* h, bool collide);
tdlb::IbmArgs ibm_args(tdlb_lattice* h, float alpha, float beta);
// Queue h's work on `s` instead of its own stream (batches share one).
void borrow_stream(tdlb_lattice* h, cudaStream_t s);
// Undo borrow_stream: h's work goes to its own stream again.
void return_stream(tdlb_lattice* h);
// Work other than the step loop's own is about to be queued on `stream`: the
// next outer launch of a split step waits for it (every entry point other than
// the step loop's calls it).
inline void fence(tdlb_lattice* h) { h->bulk_ok = false; }
// A forcing pass of the resident markers has been queued.
void note_pass(tdlb_lattice* h, float beta);
// The handle's device scratch, at least `bytes` long (kept for the next call).
cudaError_t scratch(tdlb_lattice* h, size_t bytes, char** out);
// Memory for the zone, where the handle's steps may use one; without it they
// do not split.
void reserve_zone(tdlb_lattice* h);
// Free the zone's arrays (the lattice changed size).
void drop_zone(tdlb_lattice* h);
// Remove the residual box (a tank joining a batch, whose step kernel keeps
// none), or set its residuals to zero (after the planes were written
// without them).
void drop_residual_box(tdlb_lattice* h);
void clear_residual_box(tdlb_lattice* h);
}  // namespace tdlb_rt
