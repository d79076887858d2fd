// Host runtime and C ABI (include/tdlb_b200.h) of the B200 lattice Boltzmann
// time step: device memory, the marker scheduler, launch sequencing and
// state bookkeeping. Kernels live in step_kernels.cu and ibm_kernels.cu.
#include "tdlb_b200.h"
#include "tdlb_kernels.cuh"
#include "tdlb_runtime.hpp"
#include "tdlb_geometry.hpp"

#include <nlohmann/json.hpp>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <stdexcept>
#include <string>
#include <vector>

using tdlb::Dims;
using tdlb::Planes;

namespace {

thread_local std::string g_create_error = "no error";

struct Fail {
    int code;
    std::string msg;
};

#define TDLB_CK(call)                                                                          \
    do {                                                                                       \
        cudaError_t e_ = (call);                                                               \
        if (e_ != cudaSuccess)                                                                 \
            throw Fail{TDLB_ECUDA, tdlb_rt::error_text(#call, e_)};                            \
    } while (0)

long long round_up(long long a, long long m) { return (a + m - 1) / m * m; }

}  // namespace

#include "tdlb_handle.hpp"

namespace {

void release(tdlb_lattice* h) {
    if (!h) return;
    cudaSetDevice(h->device);
    cudaFree(h->block);
    cudaFree(h->d_markers);
    cudaFree(h->d_markers_in);
    cudaFree(h->d_sched_tmp);
    cudaFree(h->d_sched);
    cudaFree(h->d_level_ptr);
    cudaFree(h->d_plane_lv0);
    cudaFree(h->d_plane_lv1);
    cudaFree(h->d_blade_planes);
    cudaFree(h->d_cell_e);
    cudaFree(h->d_plane_cell);
    cudaFree(h->d_prep);
    cudaFree(h->d_cell_m);
    cudaFree(h->d_cell_F);
    cudaFree(h->d_tail);
    cudaFree(h->d_sums);
    cudaFree(h->d_mask_static);
    cudaFree(h->d_plane_list);
    cudaFree(h->d_exclude);
    tdlb_rt::drop_zone(h);
    cudaFree(h->d_box_list);
    cudaFree(h->d_box_except);
    cudaFree(h->d_scratch);
    for (cudaEvent_t e : h->tev) cudaEventDestroy(e);
    if (h->side) cudaStreamDestroy(h->side);
    if (h->bulk) cudaStreamDestroy(h->bulk);
    if (h->ev_fork) cudaEventDestroy(h->ev_fork);
    if (h->ev_join) cudaEventDestroy(h->ev_join);
    if (h->ev_outer) cudaEventDestroy(h->ev_outer);
    if (h->ev_inner) cudaEventDestroy(h->ev_inner);
    if (h->ev_fence) cudaEventDestroy(h->ev_fence);
    cudaFree(h->d_red);
    cudaFree(h->imp_block);
    cudaFree(h->d_res[0]);
    cudaFree(h->d_res[1]);
    for (auto& st : h->pin) {
        cudaFreeHost(st.p);
        if (st.ev) cudaEventDestroy(st.ev);
    }
    if (h->own_stream) cudaStreamDestroy(h->own_stream);
    else if (h->stream) cudaStreamDestroy(h->stream);
}

void validate_config(const tdlb_config& c) {
    if (c.x < 1 || c.y < 1 || c.z < 1) throw Fail{TDLB_EINVAL, "grid extents must be >= 1"};
    if (c.x > 32767 || c.y > 32767 || c.z > 32767) throw Fail{TDLB_EINVAL, "grid extent above 32767"};
    if (c.streaming != TDLB_STREAMING_SIMPLE && c.streaming != TDLB_STREAMING_ESOTWIST)
        throw Fail{TDLB_EINVAL, "streaming must be Simple (0) or Esotwist (1)"};
    if (c.storage < TDLB_STORAGE_FP32 || c.storage > TDLB_STORAGE_BF16)
        throw Fail{TDLB_EINVAL, "storage must be FP32 (0), FP16 (1) or BF16 (2)"};
    if (c.storage != TDLB_STORAGE_FP32 && !(c.initialRho > 0.0))
        throw Fail{TDLB_EINVAL, "16-bit storage needs initialRho > 0 (deviations are taken from it)"};
    if (!(c.nu >= 0.0) || !std::isfinite(c.nu)) throw Fail{TDLB_EINVAL, "nu must be finite and >= 0"};
}

tdlb_lattice* build(const tdlb_config& c, int device) {
    validate_config(c);
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
        throw Fail{TDLB_ECUDA, "no CUDA device available (this library has no CPU path)"};
    if (device < 0 || device >= ndev) throw Fail{TDLB_EINVAL, "device index out of range"};
    int major = 0, minor = 0;   // (the whole cudaDeviceProp takes 2 to 10 ms to fill)
    TDLB_CK(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device));
    TDLB_CK(cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, device));
    if (major < 10) throw Fail{TDLB_ECUDA, "this library is built for sm_100a (B200); device is sm_" +
                                               std::to_string(major) + std::to_string(minor)};
    auto* h = new tdlb_lattice();
    try {
        h->cfg = c;
        h->device = device;
        h->vec = tdlb_rt::default_cells_per_thread(c);
        h->err.reserve(512);
        TDLB_CK(cudaSetDevice(device));
        // the forcing pass is the latency-bound path of a split step: its
        // streams get the highest priority, so its blocks are scheduled ahead
        // of the outer launch's as SMs free up
        int prio_lo = 0, prio_hi = 0;
        TDLB_CK(cudaDeviceGetStreamPriorityRange(&prio_lo, &prio_hi));
        TDLB_CK(cudaStreamCreateWithPriority(&h->stream, cudaStreamNonBlocking, prio_hi));
        TDLB_CK(cudaStreamCreateWithPriority(&h->side, cudaStreamNonBlocking, prio_hi));
        TDLB_CK(cudaStreamCreateWithPriority(&h->bulk, cudaStreamNonBlocking, prio_lo));
        TDLB_CK(cudaEventCreateWithFlags(&h->ev_fork, cudaEventDisableTiming));
        TDLB_CK(cudaEventCreateWithFlags(&h->ev_join, cudaEventDisableTiming));
        TDLB_CK(cudaEventCreateWithFlags(&h->ev_outer, cudaEventDisableTiming));
        TDLB_CK(cudaEventCreateWithFlags(&h->ev_inner, cudaEventDisableTiming));
        TDLB_CK(cudaEventCreateWithFlags(&h->ev_fence, cudaEventDisableTiming));
        Dims& g = h->g;
        g = tdlb::make_dims((int)c.x, (int)c.y, (int)c.z);
        h->mask_words = round_up(g.rows() * g.jw, 64);
        // (the limit that the 16-element row granule along z gave)
        if (c.x * c.y * round_up(c.z, 16) >= tdlb::kMaxPlane || g.rows() * g.jp >= tdlb::kMaxPlane)
            throw Fail{TDLB_EINVAL, "lattice too large: one population plane must stay below 2^31 elements"};
        h->cp = tdlb::make_collide_params(c.nu, c.cs0, c.g3);
        tdlb::set_rest(h->cp, c.initialRho);

        const tdlb_rt::LatticeBlock lb = tdlb_rt::lattice_block(g, h->mask_words, h->esz(), c.streaming == TDLB_STREAMING_SIMPLE);
        size_t free_b = 0, total_b = 0;
        TDLB_CK(cudaMemGetInfo(&free_b, &total_b));
        if (lb.bytes > free_b) throw Fail{TDLB_ENOMEM, "lattice needs " + std::to_string(lb.bytes) + " B, " +
                                                           std::to_string(free_b) + " B free on device"};
        TDLB_CK(cudaMalloc(&h->block, lb.bytes));
        lb.place(h);
        TDLB_CK(cudaMemsetAsync(h->block, 0, lb.bytes, h->stream));
        TDLB_CK(cudaStreamSynchronize(h->stream));
    } catch (...) {
        release(h);
        delete h;
        throw;
    }
    return h;
}

// Reference JSON -> tdlb_config (main.cpp:135-164 reads these sections).
tdlb_config config_from_json(const char* text) {
    nlohmann::json j;
    try {
        j = nlohmann::json::parse(text);
    } catch (const std::exception& e) {
        throw Fail{TDLB_EJSON, std::string("input JSON: ") + e.what()};
    }
    tdlb_config c{};
    try {
        const auto& grid = j.at("GridParams");
        const auto& flow = j.at("FlowParams");
        c.x = (int64_t)grid.at("x").get<uint64_t>();
        c.y = (int64_t)grid.at("y").get<uint64_t>();
        c.z = (int64_t)grid.at("z").get<uint64_t>();
        const int64_t ghost = (int64_t)grid.value("multiStep", (uint64_t)1);
        if (ghost != 1) throw Fail{TDLB_EINVAL, "GridParams.multiStep (ghost width) must be 1"};
        c.initialRho = flow.at("initialRho").get<double>();
        c.nu = flow.at("nu").get<double>();
        c.cs0 = flow.at("cs0").get<double>();
        c.g3 = flow.at("g3").get<double>();
        c.alpha = flow.at("alpha").get<double>();
        c.beta = flow.at("beta").get<double>();
        c.useLES = flow.at("useLES").get<bool>() ? 1 : 0;
        // main.cpp:242-256: "Simple" selects Simple, anything else Esotwist
        c.streaming = flow.at("streaming").get<std::string>() == "Simple" ? TDLB_STREAMING_SIMPLE : TDLB_STREAMING_ESOTWIST;
        // nu as the file gives it: main.cpp constructs the ComputeUnit from
        // its FlowParams (:242-256) before calcNuAndRe_m (:275) sets nu in
        // main's own copy, so the reference's unit keeps the file's value.
        // The FlowParams fields are float in the reference (useQVecPrecision).
        c.initialRho = (double)(float)c.initialRho;
        c.nu = (double)(float)c.nu;
        c.cs0 = (double)(float)c.cs0;
        c.g3 = (double)(float)c.g3;
        c.alpha = (double)(float)c.alpha;
        c.beta = (double)(float)c.beta;
    } catch (const Fail&) {
        throw;
    } catch (const std::exception& e) {
        throw Fail{TDLB_EJSON, std::string("input JSON: ") + e.what()};
    }
    c.storage = TDLB_STORAGE_FP32;
    return c;
}

// FENCE: what `fn` queues or changes may concern the populations, so the next
// outer launch of a split step waits for it; the step loop's own calls
// (collision, forcing_resident, rotate_impeller, set_rotating_markers, step, the
// impeller load) touch nothing that launch reads or writes.
template <bool FENCE = true, typename F>
int guarded(tdlb_lattice* h, F&& fn) {
    if (!h) return TDLB_EINVAL;
    try {
        cudaSetDevice(h->device);
        if (FENCE) tdlb_rt::fence(h);
        fn();
        return TDLB_OK;
    } catch (const Fail& f) {
        h->err = f.msg;
        return f.code;
    } catch (const std::bad_alloc&) {
        h->err = "host allocation failed";
        return TDLB_ENOMEM;
    } catch (const std::exception& e) {
        h->err = e.what();
        return TDLB_EINVAL;
    }
}

void require_init(tdlb_lattice* h) {
    if (!h->initialised) throw Fail{TDLB_ESTATE, "call tdlb_initialise() first"};
}

tdlb::StepArgs step_args(tdlb_lattice* h, bool collide) {
    tdlb::StepArgs a{};
    a.A = h->planes(h->state_buf());
    if (h->cfg.streaming == TDLB_STREAMING_SIMPLE) a.B = h->planes(h->other_buf());
    a.Nu = h->Nu;
    a.F = reinterpret_cast<const float4*>(h->F);
    a.mask = h->mask_cur();
    a.g = h->g;
    a.p = h->cp;
    a.les = h->cfg.useLES;
    a.from_moments = h->holds_moments ? 1 : 0;
    a.collide = collide ? 1 : 0;
    a.even = h->even ? 1 : 0;
    a.vec = tdlb::vector_width(h->g, h->vec);
    a.l2_prefetch = h->l2_prefetch;
    a.storage = h->cfg.storage;
    // residual box (16-bit storage): Simple reads the state buffer's
    // residuals and writes the other buffer's; Esotwist updates its one set
    a.rr = h->rbox(h->state_index());
    a.rw = h->cfg.streaming == TDLB_STREAMING_SIMPLE ? h->rbox(1 - h->state_index()) : a.rr;
    return a;
}

// ---------------------------------------------------------------------------
// Split steps.
//
// The forcing pass reads and writes only cells inside the stencils of the
// markers, and the step reads F only there. The "zone" (zone.cu) is the set of
// flag words (32 cells of a row) that hold every stencil cell of the resident
// markers at any impeller angle and, for Esotwist, their 26 neighbours. A step
// then runs as
//   bulk:   wait(inner words of step s-1), outer words of step s
//   stream: forcing pass s-1, inner words of step s, wait(outer words of step
//           s), forcing pass s
// so forcing pass s-1 and the inner words run beside the outer words of step s:
// those cells neither read F nor share a population location with a stencil
// cell, and every cell computes exactly what the unsplit step computes. With
// rows along j the zone of a stirred tank is whole rows (3 to 5 % of a 400^3
// tank), so the outer launch is the full launch in all but the rows it drops,
// and a step takes as long as the longer of the two streams. The outer launch
// follows the inner words of the step before it, not all of `stream`: what a
// caller queues there is not waited for, unless a call that fences (tdlb_join)
// comes first.
// ---------------------------------------------------------------------------

// Every stencil cell of markers [0, n) is set in `core`.
bool stencils_inside(const Dims& g, const tdlb_marker* m, size_t n, const std::vector<uint32_t>& core) {
    for (size_t q = 0; q < n; q++) {
        int st[9];
        tdlb::MarkerSchedule::stencil(reinterpret_cast<const tdlb::Marker*>(m)[q], g.nx, g.nz, st);
        const int j = (int)m[q].j;
        for (int c = 0; c < 9; c++)
            if (!((core[(size_t)g.word(st[c] / g.nz, j, st[c] % g.nz)] >> (j & 31)) & 1u)) return false;
    }
    return true;
}

// Host blades (tdlb_set_rotating_markers) against the zone's stencil cells.
bool blades_in_zone(tdlb_lattice* h) {
    const size_t n1 = (size_t)(h->n_markers - h->n0);
    if (n1 == 0 || h->rot_device) return true;   // device rotation stays inside the zone's annuli
    if (h->h_zone_core.empty()) {
        h->h_zone_core.resize((size_t)(h->g.rows() * h->g.jw));
        TDLB_CK(cudaMemcpyAsync(h->h_zone_core.data(), h->d_zone_core, h->h_zone_core.size() * sizeof(uint32_t),
                                cudaMemcpyDeviceToHost, h->stream));
        TDLB_CK(cudaStreamSynchronize(h->stream));
    }
    return stencils_inside(h->g, h->h_blades.data(), n1, h->h_zone_core);
}

void build_zone(tdlb_lattice* h) {
    TDLB_CK(cudaStreamSynchronize(h->stream));   // no launch still reads the old zone
    const Dims& g = h->g;
    const long long nw = g.rows() * g.jw;
    h->zone_gen = ~0u;
    h->h_zone_core.clear();
    const int n1 = h->n_markers - h->n0;
    if (n1 > 0) {
        // Blades turn about (ci, ck). A blade marker at radius r rounds to the
        // nearest cell, and its stencil cells lie within 1.5 cells of that
        // position per axis, so within r +- 2.13 of the axis: plane by plane,
        // the annulus between the smallest and the largest blade radius
        // widened by 3 cells. (Blades that the host has set since are held
        // against it, blades_in_zone.)
        std::vector<double2> ring((size_t)g.ny, make_double2(1e300, -1.0));
        for (int q = 0; q < n1; q++) {
            const double r = std::sqrt(h->h_rot_xz[2 * q] * h->h_rot_xz[2 * q] + h->h_rot_xz[2 * q + 1] * h->h_rot_xz[2 * q + 1]);
            double2& p = ring[(size_t)h->h_rot_j[(size_t)q]];
            p.x = std::min(p.x, r - 3.0);
            p.y = std::max(p.y, r + 3.0);
        }
        TDLB_CK(cudaMemcpy(h->d_zone_ring, ring.data(), ring.size() * sizeof(double2), cudaMemcpyHostToDevice));
    }
    TDLB_CK(tdlb::launch_zone_core(g, h->d_mask_static, n1 > 0 ? h->d_zone_ring : nullptr, h->rot_ci, h->rot_ck, h->d_zone_core,
                                   h->stream));
    TDLB_CK(tdlb::launch_zone_words(g, h->d_zone_core, h->cfg.streaming == TDLB_STREAMING_ESOTWIST, h->d_zone_skip, h->stream));
    TDLB_CK(tdlb::launch_zone_box(g, h->d_box_list, h->n_box, nullptr, h->d_zone_skip, h->stream));
    h->h_zone_skip.resize((size_t)nw);
    TDLB_CK(cudaMemcpyAsync(h->h_zone_skip.data(), h->d_zone_skip, (size_t)nw, cudaMemcpyDeviceToHost, h->stream));
    TDLB_CK(cudaStreamSynchronize(h->stream));
    std::vector<int> words;
    long long inner_cells = 0;
    for (long long w = 0; w < nw; w++)
        if (h->h_zone_skip[(size_t)w]) {
            words.push_back((int)w);
            inner_cells += std::min(32, g.ny - (int)(w % g.jw) * 32);
        }
    if (!words.empty())
        TDLB_CK(cudaMemcpy(h->d_zone_words, words.data(), words.size() * sizeof(int), cudaMemcpyHostToDevice));
    h->n_zone = (int)words.size();
    h->n_outer = (int)(nw - h->n_zone);
    h->zone_small = (double)inner_cells <= 0.6 * (double)g.cells();
    h->zone_ok = blades_in_zone(h);
    h->zone_gen = h->marker_gen;
    h->zone_box_gen = h->box_gen;
}

// The zone of the resident markers can be built.
bool zone_known(tdlb_lattice* h) {
    if (!h->markers_set || !h->resident || !h->zone_block) return false;
    const size_t n1 = (size_t)(h->n_markers - h->n0);
    return n1 == 0 || (h->impeller_begin >= 0 && h->h_rot_xz.size() == 2 * n1);
}

// The zone (when there is one for the resident markers) holds every cell that
// the last forcing pass touched: F is zero outside it. The markers may have been
// replaced since that pass, and the pass's blades by others.
bool force_in_zone(const tdlb_lattice* h) {
    return !h->forced || (h->force_gen == h->marker_gen && h->force_blades_in);
}

// A zone is planned (a wait and a pass over the flag words, 1.4 ms at 400^3) once
// the list has been through this many passes, for lattices whose steps were not
// asked to split: markers set anew with every step, before the collision or after
// it, go through one.
constexpr int kSettledPasses = 2;

// The resident markers' zone is there, or is built now.
bool zone_built(tdlb_lattice* h, bool may_build) {
    if (!zone_known(h)) return false;
    if (h->zone_gen == h->marker_gen && h->zone_box_gen == h->box_gen) return true;
    if (!may_build || (h->overlap <= 0 && h->list_passes < kSettledPasses)) return false;
    build_zone(h);
    return true;
}

// The coming step may leave F out of the words outside the zone.
bool zone_serves(tdlb_lattice* h, bool may_build) {
    if (h->forced && h->force_gen != h->marker_gen) return false;   // (and no zone is built for such a step)
    return zone_built(h, may_build) && h->zone_ok && force_in_zone(h);
}

// Smallest lattice whose steps split unasked.
constexpr long long kAutoSplitCells = 1 << 19;

// The lattice's steps may run split, whatever its markers.
bool split_wanted(const tdlb_lattice* h) {
    if (!h->overlap || h->own_stream) return false;
    if (h->overlap < 0 && (h->stream_taken || h->g.cells() < kAutoSplitCells)) return false;
    return h->cfg.storage != TDLB_STORAGE_FP32 || tdlb::vector_width(h->g, h->vec) == 1;
}

// A zone covering most of the lattice leaves little to overlap with.
bool zone_pays(const tdlb_lattice* h) { return h->zone_small || h->overlap == 2; }

bool under_capture(tdlb_lattice* h) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(h->stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone;
}

// Queue one step-kernel launch, bracketed by timing events when enabled.
template <typename L>
void timed_launch(tdlb_lattice* h, cudaStream_t st, L&& launch) {
    h->launches++;
    if (!h->timing) {
        TDLB_CK(launch());
        return;
    }
    cudaEvent_t a = nullptr, b = nullptr;
    TDLB_CK(cudaEventCreate(&a));
    if (cudaEventCreate(&b) != cudaSuccess) {
        cudaEventDestroy(a);
        throw Fail{TDLB_ECUDA, "cudaEventCreate failed"};
    }
    h->tev.push_back(a);
    h->tev.push_back(b);
    TDLB_CK(cudaEventRecord(a, st));
    TDLB_CK(launch());
    TDLB_CK(cudaEventRecord(b, st));
}

void run_step(tdlb_lattice* h, bool collide) {
    tdlb::StepArgs a = step_args(h, collide);
    const bool simple = h->cfg.streaming == TDLB_STREAMING_SIMPLE;
    auto launch = [&](const tdlb::StepArgs& x, cudaStream_t st) {
        return simple ? tdlb::launch_step_simple(x, st) : tdlb::launch_step_esotwist(x, st);
    };
    const bool boxed = a.rr.on();
    // a captured step stays on the captured stream and its own side stream, and
    // takes the zone as it is
    const bool wanted = collide && !h->holds_moments && split_wanted(h);
    const bool captured = (wanted || boxed) && under_capture(h);
    const bool zone = ((wanted && !captured) || boxed) && zone_serves(h, !captured);
    const bool split = wanted && !captured && zone && zone_pays(h);
    // 1: outer words, 2: inner words (or every word) without the box's cells
    auto part = [&](int which, cudaStream_t st, bool every = false) {
        tdlb::StepArgs x = a;
        x.part = which;
        x.zone.skip = h->d_zone_skip;
        x.zone.words = every ? nullptr : h->d_zone_words;
        x.zone.count = every ? (int)(h->g.rows() * h->g.jw) : h->n_zone;
        x.zone.except = boxed ? h->d_box_except : nullptr;
        if ((which == 1 ? h->n_outer : x.zone.count) > 0) timed_launch(h, st, [&] { return launch(x, st); });
    };
    auto box = [&] {
        a.box_cells = h->d_box_list;
        a.n_box = h->n_box;
        if (h->n_box > 0) timed_launch(h, h->stream, [&] { return tdlb::launch_box(a, simple, h->stream); });
    };
    if (split) {
        if (!h->bulk_ok) TDLB_CK(cudaEventRecord(h->ev_fence, h->stream));
        TDLB_CK(cudaStreamWaitEvent(h->bulk, h->bulk_ok ? h->ev_inner : h->ev_fence, 0));
        part(1, h->bulk);
        TDLB_CK(cudaEventRecord(h->ev_outer, h->bulk));
        if (boxed) box();
        part(2, h->stream);
        TDLB_CK(cudaEventRecord(h->ev_inner, h->stream));
        TDLB_CK(cudaStreamWaitEvent(h->stream, h->ev_outer, 0));
        h->bulk_ok = true;
    } else {
        tdlb_rt::fence(h);
        if (boxed) {
            // the box's cells are left out of the plain launches: the outer
            // words and the inner ones, or one over every word without a zone
            if (zone) part(1, h->stream);
            box();
            part(2, h->stream, !zone);
        } else {
            timed_launch(h, h->stream, [&] { return launch(a, h->stream); });
        }
    }
    if (simple) h->cur ^= 1;
    else h->even = !h->even;   // StreamingEsoteric.hpp:15-18
    h->holds_moments = false;
}

tdlb::IbmArgs ibm_args(tdlb_lattice* h, float alpha, float beta);

void validate_markers(const Dims& g, const tdlb_marker* m, size_t n, size_t base) {
    for (size_t q = 0; q < n; q++) {
        if (m[q].i < 0 || m[q].i >= g.nx || m[q].j < 0 || m[q].j >= g.ny || m[q].k < 0 || m[q].k >= g.nz) {
            char buf[160];
            std::snprintf(buf, sizeof buf, "marker %zu at (%lld,%lld,%lld) outside the %dx%dx%d interior", base + q,
                          (long long)m[q].i, (long long)m[q].j, (long long)m[q].k, g.nx, g.ny, g.nz);
            throw Fail{TDLB_EINVAL, buf};
        }
    }
}

// Grow the level-pointer array, keeping its contents (the first segment's
// levels stay valid when only the blade schedule grows).
void ensure_level_cap(tdlb_lattice* h, long long need) {
    if (need <= h->level_cap && h->d_level_ptr) return;
    TDLB_CK(cudaStreamSynchronize(h->stream));
    const long long cap = std::max<long long>(round_up(need * 2, 1024), 1024);
    int* p = nullptr;
    TDLB_CK(cudaMalloc(&p, cap * sizeof(int)));
    if (h->d_level_ptr) {
        const cudaError_t e = cudaMemcpy(p, h->d_level_ptr, (size_t)h->level_cap * sizeof(int), cudaMemcpyDeviceToDevice);
        if (e != cudaSuccess) {
            cudaFree(p);
            TDLB_CK(e);
        }
        cudaFree(h->d_level_ptr);
    }
    h->d_level_ptr = p;
    h->level_cap = cap;
}

// The planes whose second segment (blades) has levels, for the blade launch
// of the forcing pass, and its shared memory; uploaded when they change.
void update_blade_planes(tdlb_lattice* h) {
    const Dims& g = h->g;
    const auto& lv = h->seg1.plane_lv;
    const auto& lp = h->seg1.level_ptr;
    const int L0 = h->n_level0;
    std::vector<int> planes;
    int words = 0;
    h->blade_max = 0;
    for (int j = 0; j < g.ny; j++) {
        if (lv[(size_t)j] == lv[(size_t)j + 1]) continue;
        planes.push_back(j);
        // the level ranges are global level indices; seg1's level_ptr starts at level L0
        const int nb = lp[(size_t)(lv[(size_t)j + 1] - L0)] - lp[(size_t)(lv[(size_t)j] - L0)];
        words = std::max(words, tdlb::blade_table_words(nb));
        h->blade_max = std::max(h->blade_max, nb);
    }
    words = std::min(words, 220 * 1024 / 4);   // a plane beyond this walks its blades on global memory
    if (planes != h->h_blade_planes) {
        if (!h->d_blade_planes) TDLB_CK(cudaMalloc(&h->d_blade_planes, (size_t)std::max(g.ny, 1) * sizeof(int)));
        h->h_blade_planes = planes;
        if (!planes.empty())
            TDLB_CK(cudaMemcpyAsync(h->d_blade_planes, h->h_blade_planes.data(), planes.size() * sizeof(int),
                                    cudaMemcpyHostToDevice, h->stream));
        h->n_blade = (int)planes.size();
    }
    if (words > h->blade_words) TDLB_CK(tdlb::ibm_prepare_blades(words));
    h->blade_words = std::max(h->blade_words, words);
}

// Schedule of the second segment (h_blades), slots n0.., levels n_level0...
void build_blades(tdlb_lattice* h, const double* rot_xz) {
    const Dims& g = h->g;
    h->seg1.build(reinterpret_cast<const tdlb::Marker*>(h->h_blades.data()), 0, (int)h->h_blades.size(), g.nx, g.ny, g.nz,
                  h->n0, h->n_level0, rot_xz);
    for (int& q : h->seg1.order) q += h->n0;   // list indices
}

// Device copy of the second segment's schedule (slots n0.., levels L0..).
void upload_seg1(tdlb_lattice* h) {
    const Dims& g = h->g;
    update_blade_planes(h);
    const int L0 = h->n_level0;
    ensure_level_cap(h, (long long)L0 + h->seg1.nlevels + 1);
    const int n1 = h->n_markers - h->n0;
    if (n1) TDLB_CK(cudaMemcpyAsync(h->d_sched + h->n0, h->seg1.order.data(), (size_t)n1 * sizeof(int),
                                    cudaMemcpyHostToDevice, h->stream));
    TDLB_CK(cudaMemcpyAsync(h->d_level_ptr + L0, h->seg1.level_ptr.data(), h->seg1.level_ptr.size() * sizeof(int),
                            cudaMemcpyHostToDevice, h->stream));
    TDLB_CK(cudaMemcpyAsync(h->d_plane_lv1, h->seg1.plane_lv.data(), (size_t)(g.ny + 1) * sizeof(int),
                            cudaMemcpyHostToDevice, h->stream));
}

// Grow a device buffer to at least `need` elements (contents not kept; the
// stream's work is waited for by the free).
template <typename T>
void grow(T*& p, long long& cap, long long need, long long per) {
    if (need <= cap && p) return;
    cudaFree(p);
    p = nullptr;
    cap = 0;
    const long long n = round_up(need + need / 8, 1024);
    TDLB_CK(cudaMalloc(&p, (size_t)(n * per) * sizeof(T)));
    cap = n;
}

// What the host knows of the first segment's cells: the planes' ranges, the
// launches' shapes and tiles.
void plan_planes(tdlb_lattice* h, const int* count) {
    const Dims& g = h->g;
    h->plane_cell.assign((size_t)g.ny + 1, 0);
    for (int j = 0; j < g.ny; j++) h->plane_cell[(size_t)j + 1] = h->plane_cell[(size_t)j] + count[j];
    h->ncell = h->plane_cell[(size_t)g.ny];
    // F tiles of the ordinary planes' launch: up to 6144 cells (72 KB) of
    // shared memory; the tile is sized for the most crowded ordinary plane, at
    // least 4608 cells. Planes with more cells (an impeller disk) go to a
    // second, 512-thread launch with a tile for the largest of them (global
    // memory beyond the 227 KB shared-memory limit).
    int typical = 0;
    for (int j = 0; j < g.ny; j++)
        if (count[j] <= 6144) typical = std::max(typical, count[j]);
    const int small_cap = std::max(4608, round_up(typical, 64) > 6144 ? 6144 : (int)round_up(typical, 64));
    std::vector<int> small, big;
    h->max_cells = h->max_big = 0;
    for (int j = 0; j < g.ny; j++) {
        if (count[j] > small_cap) { big.push_back(j); h->max_big = std::max(h->max_big, count[j]); }
        else { small.push_back(j); h->max_cells = std::max(h->max_cells, count[j]); }
    }
    h->smem_cells = small_cap;
    h->n_small = (int)small.size();
    h->n_big = (int)big.size();
    h->big_tile_cells = tdlb::big_bulk_bytes(h->max_big) <= 220 * 1024 ? h->max_big : 0;
    TDLB_CK(tdlb::ibm_prepare_smem(h->smem_cells, tdlb::big_bulk_bytes(h->big_tile_cells)));
    small.insert(small.end(), big.begin(), big.end());
    if (!h->d_plane_list) TDLB_CK(cudaMalloc(&h->d_plane_list, (size_t)g.ny * sizeof(int)));
    TDLB_CK(cudaMemcpyAsync(h->d_plane_list, small.data(), (size_t)g.ny * sizeof(int), cudaMemcpyHostToDevice, h->stream));
    if (!h->d_plane_cell) TDLB_CK(cudaMalloc(&h->d_plane_cell, (size_t)(g.ny + 1) * sizeof(int)));
    TDLB_CK(cudaMemcpyAsync(h->d_plane_cell, h->plane_cell.data(), (size_t)(g.ny + 1) * sizeof(int), cudaMemcpyHostToDevice,
                            h->stream));
    h->h_plane_list = std::move(small);
    // 16 elements of padding: the spread's bulk copies and L2 prefetches
    // round a plane's cell range out to 16-byte boundaries
    if (h->ncell + 16 > h->cell_cap || !h->d_cell_e) {
        h->cell_cap = 0;   // until all three are there
        long long c1 = 0, c2 = 0, c3 = 0;
        grow(h->d_cell_e, c1, h->ncell + 16, 1);
        grow(h->d_cell_m, c2, h->ncell + 16, 4);
        grow(h->d_cell_F, c3, h->ncell + 16, 3);
        h->cell_cap = c1;
    }
}

// The first segment scheduled by the host: lists whose levels the device gave
// up on (schedule.cu). `m` is the list, already in d_markers.
void schedule_on_host(tdlb_lattice* h, const tdlb_marker* m, size_t n0) {
    const Dims& g = h->g;
    const auto* mk = reinterpret_cast<const tdlb::Marker*>(m);
    tdlb::MarkerSchedule seg;
    seg.build(mk, 0, (int)n0, g.nx, g.ny, g.nz, 0, 0);
    tdlb::CellList cells;
    cells.build(mk, seg, g);
    h->n_level0 = seg.nlevels;
    ensure_level_cap(h, (long long)seg.nlevels + 1);
    TDLB_CK(cudaMemcpyAsync(h->d_sched, seg.order.data(), n0 * sizeof(int), cudaMemcpyHostToDevice, h->stream));
    TDLB_CK(cudaMemcpyAsync(h->d_level_ptr, seg.level_ptr.data(), seg.level_ptr.size() * sizeof(int), cudaMemcpyHostToDevice,
                            h->stream));
    TDLB_CK(cudaMemcpyAsync(h->d_plane_lv0, seg.plane_lv.data(), (size_t)(g.ny + 1) * sizeof(int), cudaMemcpyHostToDevice,
                            h->stream));
    const std::vector<int> lv1((size_t)g.ny + 1, seg.nlevels);   // an empty second segment
    TDLB_CK(cudaMemcpyAsync(h->d_plane_lv1, lv1.data(), lv1.size() * sizeof(int), cudaMemcpyHostToDevice, h->stream));
    TDLB_CK(cudaMemcpy2DAsync(h->d_prep + tdlb::PF_CELL, tdlb::PF_STRIDE * sizeof(float), cells.mcell.data(), 9 * sizeof(int),
                              9 * sizeof(int), n0, cudaMemcpyHostToDevice, h->stream));
    TDLB_CK(cudaStreamSynchronize(h->stream));   // the host vectors go
}

// Make `m[0, n)` the resident list: segment 0 = [0, n0) with exact levels,
// scheduled on the device (schedule.cu); segment 1 = [n0, n),
// rotation-invariant when rot_xz is given, scheduled here. A list with a marker
// outside the lattice leaves the resident one as it is.
void upload_markers(tdlb_lattice* h, const tdlb_marker* m, size_t n, size_t n0, const double* rot_xz) {
    if (n > 0 && !m) throw Fail{TDLB_EINVAL, "markers is NULL"};
    if (n > (size_t)0x7fffffff) throw Fail{TDLB_EINVAL, "too many markers"};
    const Dims& g = h->g;
    static_assert(sizeof(tdlb_marker) == sizeof(tdlb::Marker), "marker layout");
    // The list goes into the buffer that is not the resident one's (which stays
    // valid until the new list has been checked); the two change places with
    // every list, so each is held against its own length.
    if ((long long)n > h->marker_in_cap || !h->d_markers_in) {
        const long long cap = std::max<long long>(round_up((long long)n, 1024), std::max<long long>(h->marker_cap, 1024));
        TDLB_CK(cudaStreamSynchronize(h->stream));
        cudaFree(h->d_markers_in);
        h->d_markers_in = nullptr;
        h->marker_in_cap = 0;
        TDLB_CK(cudaMalloc(&h->d_markers_in, cap * sizeof(tdlb::Marker)));
        h->marker_in_cap = cap;
    }
    // scratch of the scheduler, one block
    const size_t ny = (size_t)g.ny, hist = tdlb::sched_hist_ints(g, (long long)n), maps = tdlb::sched_map_words(g);
    const size_t ints = 4 + hist + n0 + maps + 9 * n0 + n0 + ny + (ny + 1) + ny;
    if (ints * sizeof(int) > h->sched_tmp_bytes) {
        TDLB_CK(cudaStreamSynchronize(h->stream));
        cudaFree(h->d_sched_tmp);
        h->d_sched_tmp = nullptr;
        h->sched_tmp_bytes = 0;
        const size_t bytes = (ints + ints / 8) * sizeof(int);
        TDLB_CK(cudaMalloc(&h->d_sched_tmp, bytes));
        h->sched_tmp_bytes = bytes;
    }
    int* tmp = (int*)h->d_sched_tmp;
    auto take = [&](size_t k) { int* p = tmp; tmp += k; return p; };
    tdlb::SchedArgs a{};
    a.markers = h->d_markers_in;
    a.n = (int)n;
    a.n0 = (int)n0;
    a.g = g;
    a.info = take(4);
    a.plane_count = take(ny);
    a.plane_slot = take(ny + 1);
    a.hist = take(hist);
    a.by_plane = take(n0);
    a.maps = maps ? (unsigned*)take(maps) : nullptr;
    a.place = take(9 * n0);
    a.level_end = take(n0);
    a.levels = take(ny);
    if (n) TDLB_CK(cudaMemcpyAsync(h->d_markers_in, m, n * sizeof(tdlb::Marker), cudaMemcpyHostToDevice, h->stream));
    const int start[4] = {(int)n, 0, 0, 0};
    TDLB_CK(cudaMemcpyAsync(a.info, start, sizeof start, cudaMemcpyHostToDevice, h->stream));
    if (hist) TDLB_CK(cudaMemsetAsync(a.hist, 0, hist * sizeof(int), h->stream));
    TDLB_CK(tdlb::launch_sched_cells(a, h->stream));
    std::vector<int> got(4 + ny);
    TDLB_CK(cudaMemcpyAsync(got.data(), a.info, got.size() * sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    TDLB_CK(cudaStreamSynchronize(h->stream));
    if (got[0] < (int)n) validate_markers(g, m + got[0], 1, (size_t)got[0]);   // throws
    // the list is good: it becomes the resident one, and nothing that the handle
    // knows of the one before (its impeller, plans by generation) is its own,
    // whether the rest of this succeeds or not
    h->rot_device = false;
    h->impeller_begin = -1;
    h->marker_gen++;
    h->list_passes = 0;
    std::swap(h->d_markers, h->d_markers_in);
    std::swap(h->marker_cap, h->marker_in_cap);
    h->n_markers = (int)n;
    h->n0 = (int)n0;
    h->h_blades.assign(m + n0, m + n);
    h->markers_set = false;   // until all of this is done
    if (h->marker_cap > h->slot_cap || !h->d_sched) {
        cudaFree(h->d_sched);
        cudaFree(h->d_sums);
        h->d_sched = nullptr;
        h->d_sums = nullptr;
        h->slot_cap = 0;
        TDLB_CK(cudaMalloc(&h->d_sched, h->marker_cap * sizeof(int)));
        TDLB_CK(cudaMalloc(&h->d_sums, (size_t)3 * h->marker_cap * sizeof(float)));
        h->slot_cap = h->marker_cap;
    }
    const long long ntail = (long long)n - (long long)n0;
    if (ntail > h->tail_cap) {
        cudaFree(h->d_tail);
        h->d_tail = nullptr;
        h->tail_cap = 0;
        const long long cap = round_up(ntail, 256);
        TDLB_CK(cudaMalloc(&h->d_tail, (size_t)tdlb::TF_COUNT * cap * sizeof(float)));
        h->tail_cap = cap;
    }
    plan_planes(h, got.data() + 4);
    if ((long long)n0 > 0) grow(h->d_prep, h->prep_cap, (long long)n0 + 1, tdlb::PF_STRIDE);
    if (!h->d_mask_static) TDLB_CK(cudaMalloc(&h->d_mask_static, (size_t)h->mask_words * sizeof(uint32_t)));
    TDLB_CK(cudaMemsetAsync(h->d_mask_static, 0, (size_t)h->mask_words * sizeof(uint32_t), h->stream));
    if (!h->d_plane_lv0) TDLB_CK(cudaMalloc(&h->d_plane_lv0, (size_t)(g.ny + 1) * sizeof(int)));
    if (!h->d_plane_lv1) TDLB_CK(cudaMalloc(&h->d_plane_lv1, (size_t)(g.ny + 1) * sizeof(int)));
    ensure_level_cap(h, (long long)n + 1);   // (never more levels than markers)
    a.markers = h->d_markers;
    a.owner = (int*)h->d_cell_F;
    a.plane_cell = h->d_plane_cell;
    a.cell_e = h->d_cell_e;
    a.sched = h->d_sched;
    a.prep = h->d_prep;
    a.level_ptr = h->d_level_ptr;
    a.plane_lv0 = h->d_plane_lv0;
    a.plane_lv1 = h->d_plane_lv1;
    a.mask_static = h->d_mask_static;
    TDLB_CK(tdlb::launch_sched_levels(a, std::max(h->max_cells, h->max_big), h->ncell, h->stream));
    TDLB_CK(cudaMemcpyAsync(got.data(), a.info, 4 * sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    TDLB_CK(cudaStreamSynchronize(h->stream));
    h->n_level0 = got[2];
    if (got[1]) schedule_on_host(h, m, n0);
    if (n0) TDLB_CK(tdlb::launch_ibm_prepare(ibm_args(h, 0.f, 0.f), h->d_prep, h->stream));
    // the blades
    h->h_blade_planes.clear();
    h->n_blade = h->blade_max = 0;
    if (ntail > 0) {
        build_blades(h, rot_xz);
        upload_seg1(h);
        TDLB_CK(cudaStreamSynchronize(h->stream));   // the host vectors are read by queued copies
    }
    h->markers_set = true;
}

tdlb::IbmArgs ibm_args(tdlb_lattice* h, float alpha, float beta) {
    tdlb::IbmArgs a{};
    a.markers = h->d_markers;
    a.sched = h->d_sched;
    a.level_ptr = h->d_level_ptr;
    a.plane_lv0 = h->d_plane_lv0;
    a.plane_lv1 = h->d_plane_lv1;
    a.n = h->n_markers;
    a.n0 = h->n0;
    a.cell_e = h->d_cell_e;
    a.plane_cell = h->d_plane_cell;
    a.ncell = h->ncell;
    a.max_cells = h->max_cells;
    a.max_big = h->max_big;
    a.prep = h->d_prep;
    a.cell_m = h->d_cell_m;
    a.cell_F = h->d_cell_F;
    a.tail = h->d_tail;
    a.tail_cap = h->tail_cap;
    a.sums = h->d_sums;
    a.smem_cells = h->smem_cells;
    a.plane_list = h->d_plane_list;
    a.n_small = h->n_small;
    a.n_big = h->n_big;
    a.blade_planes = h->d_blade_planes;
    a.n_blade = h->n_blade;
    a.blade_words = h->blade_words;
    a.blade_max = h->blade_max;
    a.big_tile_cells = h->big_tile_cells;
    a.side = h->side;
    a.ev_fork = h->ev_fork;
    a.ev_join = h->ev_join;
    a.A = h->planes(h->state_buf());
    a.state_mode = h->state_mode();
    a.even = h->even ? 1 : 0;
    a.F4 = reinterpret_cast<float4*>(h->F);
    a.mask_old = h->mask_cur();
    a.mask_new = h->mask_next();
    a.mask_static = h->d_mask_static;
    a.mask_bytes = (size_t)h->mask_words * sizeof(uint32_t);
    a.g = h->g;
    a.alpha = alpha;
    a.beta = beta;
    a.storage = h->cfg.storage;
    a.p = h->cp;
    a.rbox = h->rbox(h->state_index());
    return a;
}

void run_forcing(tdlb_lattice* h, float alpha, float beta) {
    if (!h->markers_set) throw Fail{TDLB_ESTATE, "no markers set (tdlb_set_markers / tdlb_forcing)"};
    TDLB_CK(tdlb::launch_ibm(ibm_args(h, alpha, beta), h->stream));
    h->launches += 1 + (h->n_small > 0 ? 1 : 0) + (h->n_big > 0 ? 1 : 0) +
                   (h->n_blade > 0 && (h->n_big > 0 || h->blade_max > 128) ? 1 : 0);
    h->pass++;
    tdlb_rt::note_pass(h, beta);
}

void host_aos_to_planes(tdlb_lattice* h, const float* in, int npl, float* dev) {
    const Dims& g = h->g;
    std::vector<float> tmp((size_t)npl * g.plane, 0.f);
    size_t c = 0;
    for (int i = 0; i < g.nx; i++)
        for (int j = 0; j < g.ny; j++)
            for (int k = 0; k < g.nz; k++, c++) {
                const size_t e = (size_t)g.at(i, j, k);
                for (int l = 0; l < npl; l++) tmp[(size_t)l * g.plane + e] = in[c * npl + l];
            }
    TDLB_CK(cudaMemcpyAsync(dev, tmp.data(), tmp.size() * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    TDLB_CK(cudaStreamSynchronize(h->stream));
}

// The impeller's arrays, one allocation kept for the next impeller: its blades'
// offsets, the load's scratch and the impeller's slots of the resident list (the
// markers from list index `begin`), the staging of a blade upload (the blades,
// their order, at most a level each, the planes' level offsets). Made with the
// impeller, so that neither a load nor a blade upload allocates or waits. (The
// blades keep their slots while they rotate on the device; a host list of blades
// reorders them within the second segment, which is the impeller's whole.)
constexpr size_t kLoadDoubles = (size_t)tdlb::kLoadBlocks * 5 + 5 + 1;
void prepare_impeller(tdlb_lattice* h, const std::vector<double>& xz, int begin) {
    const int n = h->n_markers, groups = (n + 255) / 256;
    const size_t blades = xz.size() / 2;
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t here = at;
        at += (bytes + 255) / 256 * 256;
        return here;
    };
    const size_t o_xz = take(xz.size() * sizeof(double)), o_load = take(kLoadDoubles * sizeof(double)),
                 o_slots = take((size_t)(n - begin) * sizeof(int)), o_off = take((size_t)groups * sizeof(int)),
                 o_stage = take(blades * (sizeof(tdlb::Marker) + 2 * sizeof(int)) + (size_t)(h->g.ny + 2) * sizeof(int));
    if (at > h->imp_block_cap) {
        TDLB_CK(cudaStreamSynchronize(h->stream));
        cudaFree(h->imp_block);
        h->imp_block = nullptr;
        h->imp_block_cap = 0;
        TDLB_CK(cudaMalloc(&h->imp_block, at));
        h->imp_block_cap = at;
    }
    h->d_rot_xz = (double*)(h->imp_block + o_xz);
    h->d_load = (double*)(h->imp_block + o_load);
    h->d_imp_slots = (int*)(h->imp_block + o_slots);
    h->d_blade_stage = h->imp_block + o_stage;
    h->n_imp = n - begin;
    int* off = (int*)(h->imp_block + o_off);
    std::vector<int> count((size_t)groups);
    if (!xz.empty())
        TDLB_CK(cudaMemcpyAsync(h->d_rot_xz, xz.data(), xz.size() * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    TDLB_CK(cudaMemsetAsync(h->d_load, 0, kLoadDoubles * sizeof(double), h->stream));
    TDLB_CK(tdlb::launch_impeller_slots(h->d_sched, n, begin, off, nullptr, h->stream));
    if (n) TDLB_CK(cudaMemcpyAsync(count.data(), off, (size_t)groups * sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    TDLB_CK(cudaStreamSynchronize(h->stream));
    int sum = 0;
    for (int& c : count) {
        const int v = c;
        c = sum;
        sum += v;
    }
    if (n) TDLB_CK(cudaMemcpyAsync(off, count.data(), (size_t)groups * sizeof(int), cudaMemcpyHostToDevice, h->stream));
    TDLB_CK(tdlb::launch_impeller_slots(h->d_sched, n, begin, off, h->d_imp_slots, h->stream));
}

// ---------------------------------------------------------------------------
// Residual box of the 16-bit storage (tdlb::ResidualBox): exact deviations
// for every population location inside a box of cells.
// ---------------------------------------------------------------------------
void drop_rbox(tdlb_lattice* h) {
    cudaFree(h->d_res[0]);
    cudaFree(h->d_res[1]);
    h->d_res[0] = h->d_res[1] = nullptr;
    cudaFree(h->d_box_list);
    cudaFree(h->d_box_except);
    h->d_box_list = nullptr;
    h->d_box_except = nullptr;
    h->n_box = 0;
    h->rbox_geom = tdlb::ResidualBox{};
    h->box_gen++;
}

// The cells that the box launch of a step takes, by element, and their bits.
// Which cells these are is part of the results: the box launch's
// scalar arithmetic and the plain kernel's packed one differ
// by FP32 ulps, which 16-bit storage then rounds. They are the cells of every
// group of 32 along k (groups counted through the lines of constant (i, j),
// lines padded to 16 cells) that holds a cell near the box.
void build_box_list(tdlb_lattice* h) {
    const Dims& g = h->g;
    const tdlb::ResidualBox& b = h->rbox_geom;
    const long long line = round_up(g.nz, 16), ngroups = ((long long)g.nx * g.ny * line + 31) / 32;
    std::vector<uint8_t> hit((size_t)ngroups, 0);
    for (int i = std::max(0, b.i0 - 1); i <= std::min(g.nx - 1, b.i0 + b.bx); i++)
        for (int j = std::max(0, b.j0 - 1); j <= std::min(g.ny - 1, b.j0 + b.by); j++)
            for (int k = std::max(0, b.k0 - 1); k <= std::min(g.nz - 1, b.k0 + b.bz); k++)
                if (b.around(i, j, k)) hit[(size_t)((((long long)i * g.ny + j) * line + k) >> 5)] = 1;
    std::vector<int> list;
    // in element order; a group may reach into the lines before and after
    int j0 = b.j0 - 2, j1 = b.j0 + b.by + 2;
    if (j0 < 0 || j1 > g.ny) {
        j0 = 0;
        j1 = g.ny;
    }
    for (int i = std::max(0, b.i0 - 2); i < std::min(g.nx, b.i0 + b.bx + 2); i++)
        for (int k = 0; k < g.nz; k++)
            for (int j = j0; j < j1; j++)
                if (hit[(size_t)((((long long)i * g.ny + j) * line + k) >> 5)]) list.push_back((int)g.at(i, j, k));
    const size_t n = std::max<size_t>(list.size(), 1) * sizeof(int), bits = (size_t)(g.rows() * g.jw) * sizeof(uint32_t);
    TDLB_CK(cudaMalloc(&h->d_box_list, n));
    TDLB_CK(cudaMalloc(&h->d_box_except, bits));
    if (!list.empty())
        TDLB_CK(cudaMemcpyAsync(h->d_box_list, list.data(), list.size() * sizeof(int), cudaMemcpyHostToDevice, h->stream));
    TDLB_CK(cudaMemsetAsync(h->d_box_except, 0, bits, h->stream));
    TDLB_CK(tdlb::launch_zone_box(g, h->d_box_list, (int)list.size(), h->d_box_except, nullptr, h->stream));
    TDLB_CK(cudaStreamSynchronize(h->stream));
    h->n_box = (int)list.size();
}

// The box [i0, i1) x [j0, j1) x [k0, k1); an empty one removes the box. The
// residuals start at zero: every location holds its 16-bit value exactly,
// and steps refine the locations inside the box from then on.
void set_rbox(tdlb_lattice* h, long long i0, long long i1, long long j0, long long j1, long long k0, long long k1) {
    const Dims& g = h->g;
    if (i1 <= i0 || j1 <= j0 || k1 <= k0) {
        drop_rbox(h);
        return;
    }
    // a rejected box leaves the current one in place
    if (h->cfg.storage == TDLB_STORAGE_FP32) throw Fail{TDLB_EINVAL, "a residual box needs 16-bit storage (FP32 storage is exact)"};
    if (h->own_stream) throw Fail{TDLB_ESTATE, "a tank of a batch has no residual box"};
    // no box cell at index 0: an Esotwist location that wraps around the
    // lattice (index 0) then never lies in the box
    if (i0 < 1 || j0 < 1 || k0 < 1 || i1 > g.nx || j1 > g.ny || k1 > g.nz)
        throw Fail{TDLB_EINVAL, "the residual box must lie within [1, x) x [1, y) x [1, z)"};
    drop_rbox(h);   // (the frees wait for the launches that read the old one)
    tdlb::ResidualBox b;
    b.i0 = (int)i0; b.j0 = (int)j0; b.k0 = (int)k0;
    b.bx = (int)(i1 - i0); b.by = (int)(j1 - j0); b.bz = (int)(k1 - k0);
    b.n = (long long)b.bx * b.by * b.bz;
    const int sets = h->cfg.streaming == TDLB_STREAMING_SIMPLE ? 2 : 1;
    for (int q = 0; q < sets; q++) {
        const size_t bytes = (size_t)tdlb::NQ * (size_t)b.n * sizeof(float);
        cudaError_t e = cudaMalloc(&h->d_res[q], bytes);
        if (e != cudaSuccess) {
            drop_rbox(h);
            throw Fail{TDLB_ENOMEM, tdlb_rt::error_text("residual box", e)};
        }
        TDLB_CK(cudaMemsetAsync(h->d_res[q], 0, bytes, h->stream));
    }
    h->rbox_geom = b;
    try {
        build_box_list(h);
    } catch (...) {
        drop_rbox(h);
        throw;
    }
    h->box_gen++;
    tdlb_rt::reserve_zone(h);
}

// Residuals back to zero, after anything wrote the 16-bit planes without
// them (initialise, checkpoint read).
void clear_rbox(tdlb_lattice* h) {
    for (int q = 0; q < 2; q++)
        if (h->d_res[q])
            TDLB_CK(cudaMemsetAsync(h->d_res[q], 0, (size_t)tdlb::NQ * (size_t)h->rbox_geom.n * sizeof(float), h->stream));
}

// The impeller's swept volume with a margin of 4 cells: the blades' radius
// about the axis and their planes. There the 16-bit rounding of the stored
// deviations is what sets the velocity error against FP64 (FP32 storage in
// this volume alone brings FP16 from 2.2e-3 to about 6e-4 after 2000 steps
// of a 120^3 tank at Re 20000).
void auto_rbox(tdlb_lattice* h, const tdlb::RushtonGeom& G, const std::vector<tdlb::RotatingPolar>& pol, double rmax) {
    if (h->cfg.storage == TDLB_STORAGE_FP32 || !h->rbox_auto || h->own_stream || pol.empty()) return;
    long long jmin = pol[0].j, jmax = pol[0].j;
    for (const tdlb::RotatingPolar& p : pol) {
        jmin = std::min(jmin, p.j);
        jmax = std::max(jmax, p.j);
    }
    const double r = rmax + 4.0;
    const Dims& g = h->g;
    auto lo = [](double v) { return std::max(1LL, (long long)std::floor(v)); };
    set_rbox(h, lo(G.ci - r), std::min<long long>(g.nx, (long long)std::ceil(G.ci + r) + 1), std::max(1LL, jmin - 4),
             std::min<long long>(g.ny, jmax + 5), lo(G.ck - r), std::min<long long>(g.nz, (long long)std::ceil(G.ck + r) + 1));
}

}  // namespace

extern "C" {

int tdlb_create_config(const tdlb_config* cfg, int device, tdlb_handle* out) {
    if (!cfg || !out) {
        g_create_error = "NULL argument";
        return TDLB_EINVAL;
    }
    *out = nullptr;
    try {
        *out = build(*cfg, device);
        return TDLB_OK;
    } catch (const Fail& f) {
        g_create_error = f.msg;
        return f.code;
    } catch (const std::bad_alloc&) {
        g_create_error = "host allocation failed";
        return TDLB_ENOMEM;
    }
}

int tdlb_create(const char* params_json, int device, tdlb_handle* out) {
    if (!params_json || !out) {
        g_create_error = "NULL argument";
        return TDLB_EINVAL;
    }
    *out = nullptr;
    try {
        tdlb_config c = config_from_json(params_json);
        *out = build(c, device);
        return TDLB_OK;
    } catch (const Fail& f) {
        g_create_error = f.msg;
        return f.code;
    } catch (const std::bad_alloc&) {
        g_create_error = "host allocation failed";
        return TDLB_ENOMEM;
    }
}

int tdlb_config_from_json(const char* params_json, tdlb_config* out) {
    if (!params_json || !out) {
        g_create_error = "NULL argument";
        return TDLB_EINVAL;
    }
    try {
        *out = config_from_json(params_json);
        return TDLB_OK;
    } catch (const Fail& f) {
        g_create_error = f.msg;
        return f.code;
    }
}

int tdlb_lattice_bytes(const tdlb_config* c, int64_t* bytes) {
    if (!c || !bytes || c->x < 1 || c->y < 1 || c->z < 1) return TDLB_EINVAL;
    const long long jp = tdlb::row_pitch(c->x, c->y, c->z), jw = (jp + 31) / 32;
    const long long plane = round_up(c->x * c->z * jp, 64);
    const long long mask_words = round_up(c->x * c->z * jw, 64);
    const long long esz = c->storage == TDLB_STORAGE_FP32 ? 4 : 2;
    const long long pops = (long long)tdlb::NQ * plane * esz * (c->streaming == TDLB_STREAMING_SIMPLE ? 2 : 1);
    // fields, flags, the split steps' zone, and the marker buffers of a
    // tank-wall geometry (about 8 markers per (i, j) column at most, 360 bytes
    // each with the next list, the scheduler's scratch, their schedule,
    // stencil-cell and per-pass data)
    *bytes = pops + 5 * plane * 4 + (2 * 4 + 9) * mask_words + 8 * c->x * c->y * 360;   // F (float4) and Nu: 5 planes
    return TDLB_OK;
}

int tdlb_destroy(tdlb_handle h) {
    if (!h) return TDLB_EINVAL;
    release(h);
    delete h;
    return TDLB_OK;
}

const char* tdlb_last_error(tdlb_handle h) { return h ? h->err.c_str() : g_create_error.c_str(); }

int tdlb_initialise(tdlb_handle h, float rho) {
    return guarded(h, [&] {
        const Dims& g = h->g;
        h->cur = 0;
        h->even = true;
        h->holds_moments = true;
        h->pass = 0;
        h->forced = false;
        if (h->cfg.storage == TDLB_STORAGE_FP32) {
            TDLB_CK(tdlb::launch_fill_uniform_moments(h->planes(h->bufA), g, rho, h->stream));
        } else {
            // 16-bit storage holds populations only: the rest populations of
            // rho have the same moments (rho, 0, ..., 0) as the reference's Q
            TDLB_CK(tdlb::launch_fill_rest(h->planes(h->bufA), g.plane, rho, (float)h->cfg.initialRho, h->cfg.storage,
                                           h->cp, h->stream));
            h->holds_moments = false;
        }
        TDLB_CK(cudaMemsetAsync(h->Nu, 0, (size_t)g.plane * sizeof(float), h->stream));
        TDLB_CK(cudaMemsetAsync(h->F, 0, (size_t)4 * g.plane * sizeof(float), h->stream));
        TDLB_CK(cudaMemsetAsync(h->mask, 0, (size_t)2 * h->mask_words * sizeof(uint32_t), h->stream));
        clear_rbox(h);
        h->initialised = true;
    });
}

int tdlb_set_markers(tdlb_handle h, const tdlb_marker* markers, size_t n) {
    return guarded(h, [&] {
        upload_markers(h, markers, n, n, nullptr);
        h->resident = true;
        tdlb_rt::reserve_zone(h);
    });
}

int tdlb_forcing_resident(tdlb_handle h, float alpha, float beta) {
    return guarded<false>(h, [&] {
        require_init(h);
        run_forcing(h, alpha, beta);
    });
}

int tdlb_forcing(tdlb_handle h, const tdlb_marker* markers, size_t n, float alpha, float beta) {
    return guarded(h, [&] {
        require_init(h);
        upload_markers(h, markers, n, n, nullptr);
        h->resident = false;   // a new list every pass: no split-step zone
        run_forcing(h, alpha, beta);
    });
}

int tdlb_collision(tdlb_handle h) {
    return guarded<false>(h, [&] {
        require_init(h);
        run_step(h, true);
    });
}

int tdlb_bounce_back(tdlb_handle h) { return h ? TDLB_OK : TDLB_EINVAL; }
int tdlb_streaming_push(tdlb_handle h) { return h ? TDLB_OK : TDLB_EINVAL; }
int tdlb_moments(tdlb_handle h) { return h ? TDLB_OK : TDLB_EINVAL; }

int tdlb_step(tdlb_handle h, float alpha, float beta) {
    return guarded<false>(h, [&] {
        require_init(h);
        run_step(h, true);
        run_forcing(h, alpha, beta);
    });
}

int tdlb_get_dims(tdlb_handle h, int64_t* x, int64_t* y, int64_t* z) {
    return guarded<false>(h, [&] {
        if (x) *x = h->g.nx;
        if (y) *y = h->g.ny;
        if (z) *z = h->g.nz;
    });
}

int tdlb_get_even_step(tdlb_handle h, int* even) {
    return guarded<false>(h, [&] {
        if (!even) throw Fail{TDLB_EINVAL, "out is NULL"};
        *even = h->even ? 1 : 0;
    });
}

int tdlb_set_cells_per_thread(tdlb_handle h, int v) {
    return guarded(h, [&] {
        if (v != 1 && v != 2 && v != 4) throw Fail{TDLB_EINVAL, "cells per thread must be 1, 2 or 4"};
        h->vec = v;
        tdlb_rt::reserve_zone(h);
    });
}

int tdlb_set_l2_prefetch(tdlb_handle h, int on) {
    return guarded(h, [&] {
        if (on != 0 && on != 1) throw Fail{TDLB_EINVAL, "l2 prefetch must be 0 or 1"};
        h->l2_prefetch = on;
    });
}

int tdlb_set_overlap(tdlb_handle h, int mode) {
    return guarded(h, [&] {
        if (mode < -1 || mode > 2) throw Fail{TDLB_EINVAL, "overlap mode must be -1, 0, 1 or 2"};
        h->overlap = mode;
        tdlb_rt::reserve_zone(h);
    });
}

int tdlb_join(tdlb_handle h) {
    return guarded(h, [&] {});
}

int tdlb_read_zone(tdlb_handle h, uint8_t* flags) {
    return guarded(h, [&] {
        if (!flags) throw Fail{TDLB_EINVAL, "out is NULL"};
        if (!split_wanted(h) || !zone_built(h, true) || !h->zone_ok || !zone_pays(h))
            throw Fail{TDLB_ESTATE, "no split step (needs split steps on, resident markers that, unasked, have been through "
                                    "two forcing passes, one cell per thread with FP32 storage and, unless mode 2, inner "
                                    "words holding at most 60 % of the lattice)"};
        const Dims& g = h->g;
        size_t c = 0;
        for (int i = 0; i < g.nx; i++)
            for (int j = 0; j < g.ny; j++)
                for (int k = 0; k < g.nz; k++, c++) flags[c] = h->h_zone_skip[(size_t)g.word(i, j, k)];
    });
}

int tdlb_kernel_launches(tdlb_handle h, int64_t* n) {
    return guarded<false>(h, [&] {
        if (!n) throw Fail{TDLB_EINVAL, "out is NULL"};
        *n = (int64_t)h->launches;
    });
}

int tdlb_set_kernel_timing(tdlb_handle h, int on) {
    return guarded(h, [&] { h->timing = on != 0; });
}

int tdlb_kernel_time(tdlb_handle h, double* total_ms, int64_t* launches) {
    return guarded<false>(h, [&] {
        TDLB_CK(cudaStreamSynchronize(h->stream));
        double ms = 0.0;
        for (size_t q = 0; q + 1 < h->tev.size(); q += 2) {
            float t = 0.f;
            TDLB_CK(cudaEventElapsedTime(&t, h->tev[q], h->tev[q + 1]));
            ms += t;
        }
        const int64_t n = (int64_t)(h->tev.size() / 2);
        for (cudaEvent_t e : h->tev) cudaEventDestroy(e);
        h->tev.clear();
        if (total_ms) *total_ms = ms;
        if (launches) *launches = n;
    });
}

int tdlb_reduce_fp64(tdlb_handle h, double* out4) {
    return guarded(h, [&] {
        require_init(h);
        if (!out4) throw Fail{TDLB_EINVAL, "out is NULL"};
        if (!h->d_red) TDLB_CK(cudaMalloc(&h->d_red, (size_t)(tdlb::kReduceBlocks * 4 + 4) * sizeof(double)));
        tdlb::IbmArgs a = ibm_args(h, 0.f, 0.f);
        TDLB_CK(tdlb::launch_reduce_fp64(a, h->mask_cur(), h->d_red, h->d_red + tdlb::kReduceBlocks * 4, h->stream));
        TDLB_CK(cudaMemcpyAsync(out4, h->d_red + tdlb::kReduceBlocks * 4, 4 * sizeof(double), cudaMemcpyDeviceToHost,
                                h->stream));
        TDLB_CK(cudaStreamSynchronize(h->stream));
    });
}

int tdlb_get_stream(tdlb_handle h, void** stream) {
    return guarded<false>(h, [&] {
        if (!stream) throw Fail{TDLB_EINVAL, "out is NULL"};
        *stream = (void*)h->stream;
        if (!h->own_stream) h->stream_taken = true;
    });
}

int tdlb_synchronize(tdlb_handle h) {
    return guarded<false>(h, [&] { TDLB_CK(cudaStreamSynchronize(h->stream)); });
}

int tdlb_attach_rushton(tdlb_handle h, const tdlb_rushton* spec, double nonupdating_delta_angle, double angle,
                        double delta_angle) {
    return guarded(h, [&] {
        if (!spec) throw Fail{TDLB_EINVAL, "spec is NULL"};
        if (spec->x != h->g.nx || spec->y != h->g.ny || spec->z != h->g.nz)
            throw Fail{TDLB_EINVAL, "Rushton spec extents differ from the lattice"};
        const tdlb::RushtonGeom G = tdlb::RushtonGeom::from(*spec);
        std::vector<tdlb_marker> all = G.fixed();
        const int n_fixed = (int)all.size();
        const std::vector<tdlb_marker> nonupd = G.rotating_nonupdating(nonupdating_delta_angle);
        all.insert(all.end(), nonupd.begin(), nonupd.end());
        const size_t n0 = all.size();
        const std::vector<tdlb_marker> rot = G.rotating(angle, delta_angle);
        all.insert(all.end(), rot.begin(), rot.end());
        const std::vector<tdlb::RotatingPolar> pol = G.rotating_polar();
        std::vector<double> xz(2 * pol.size());
        double rmax = 0;
        for (size_t q = 0; q < pol.size(); q++) {
            xz[2 * q] = pol[q].x0;
            xz[2 * q + 1] = pol[q].z0;
            rmax = std::max(rmax, std::sqrt(pol[q].x0 * pol[q].x0 + pol[q].z0 * pol[q].z0));
        }
        if (G.ci - rmax < 2.0 || G.ci + rmax > h->g.nx - 3.0 || G.ck - rmax < 2.0 || G.ck + rmax > h->g.nz - 3.0)
            throw Fail{TDLB_EINVAL, "impeller does not stay 2 cells inside the lattice"};
        upload_markers(h, all.data(), all.size(), n0, xz.data());
        h->resident = true;
        h->h_rot_xz = xz;
        h->h_rot_j.assign(rot.size(), 0);
        for (size_t q = 0; q < rot.size(); q++) h->h_rot_j[q] = (int)rot[q].j;
        prepare_impeller(h, xz, n_fixed);
        h->rot_device = true;
        h->rot_ci = G.ci;
        h->rot_ck = G.ck;
        h->impeller_begin = n_fixed;
        h->rspec = *spec;
        h->angle = angle;
        h->rstep = 1;
        auto_rbox(h, G, pol, rmax);
        tdlb_rt::reserve_zone(h);
    });
}

int tdlb_set_residual_box(tdlb_handle h, int64_t i0, int64_t i1, int64_t j0, int64_t j1, int64_t k0, int64_t k1) {
    return guarded(h, [&] {
        set_rbox(h, i0, i1, j0, j1, k0, k1);
        h->rbox_auto = false;
    });
}

int tdlb_get_residual_box(tdlb_handle h, int64_t* box6) {
    return guarded<false>(h, [&] {
        if (!box6) throw Fail{TDLB_EINVAL, "box6 is NULL"};
        const tdlb::ResidualBox& b = h->rbox_geom;
        box6[0] = b.i0; box6[1] = b.i0 + b.bx;
        box6[2] = b.j0; box6[3] = b.j0 + b.by;
        box6[4] = b.k0; box6[5] = b.k0 + b.bz;
    });
}

int tdlb_rotate_impeller(tdlb_handle h, double angle, double delta_angle) {
    return guarded<false>(h, [&] {
        if (!h->rot_device) throw Fail{TDLB_ESTATE, "no impeller attached (tdlb_attach_rushton)"};
        // after the previous forcing pass, which reads the blades
        TDLB_CK(tdlb::launch_rotate_markers(h->d_rot_xz, h->d_markers + h->n0, h->n_markers - h->n0, std::cos(angle),
                                            std::sin(angle), delta_angle, h->rot_ci, h->rot_ck, h->g.nx, h->g.nz, h->stream));
        h->launches++;
        h->angle = angle;
    });
}

int tdlb_set_rotating_markers(tdlb_handle h, const tdlb_marker* markers, size_t n) {
    return guarded<false>(h, [&] {
        if (h->impeller_begin < 0) throw Fail{TDLB_ESTATE, "no impeller attached (tdlb_attach_rushton)"};
        if (n != (size_t)(h->n_markers - h->n0)) throw Fail{TDLB_EINVAL, "rotating marker count differs from the attached blades"};
        if (n && !markers) throw Fail{TDLB_EINVAL, "markers is NULL"};
        validate_markers(h->g, markers, n, (size_t)h->n0);
        // Host copies and the blade schedule for these positions; the uploads
        // go through a pinned buffer and are queued after the work already on
        // the stream (the previous forcing pass still reads the old blades),
        // so this call does not wait for the device.
        h->h_blades.assign(markers, markers + n);
        build_blades(h, nullptr);
        update_blade_planes(h);
        const int L0 = h->n_level0;
        ensure_level_cap(h, (long long)L0 + h->seg1.nlevels + 1);
        const size_t b_mk = n * sizeof(tdlb::Marker);
        const size_t b_order = n * sizeof(int);
        const size_t b_lv = h->seg1.level_ptr.size() * sizeof(int);
        const size_t b_pl = (size_t)(h->g.ny + 1) * sizeof(int);
        const size_t need = b_mk + b_order + b_lv + b_pl;
        auto& st = h->pin[h->pin_cur];
        h->pin_cur ^= 1;
        if (st.ev) TDLB_CK(cudaEventSynchronize(st.ev));   // the copies of two calls ago read this buffer
        else TDLB_CK(cudaEventCreateWithFlags(&st.ev, cudaEventDisableTiming));
        if (need > st.cap) {
            cudaFreeHost(st.p);
            st.p = nullptr;
            st.cap = 0;
            TDLB_CK(cudaHostAlloc((void**)&st.p, need, cudaHostAllocDefault));
            st.cap = need;
        }
        char* q = st.p;
        std::memcpy(q, markers, b_mk);
        std::memcpy(q + b_mk, h->seg1.order.data(), b_order);
        std::memcpy(q + b_mk + b_order, h->seg1.level_ptr.data(), b_lv);
        std::memcpy(q + b_mk + b_order + b_lv, h->seg1.plane_lv.data(), b_pl);
        // one copy and a launch that puts the four parts in their places (four
        // copies of a few KB are four trips)
        TDLB_CK(cudaMemcpyAsync(h->d_blade_stage, q, need, cudaMemcpyHostToDevice, h->stream));
        TDLB_CK(cudaEventRecord(st.ev, h->stream));
        TDLB_CK(tdlb::launch_place_blades((const int*)h->d_blade_stage, h->d_markers + h->n0, (int)n, h->d_sched + h->n0,
                                          h->d_level_ptr + L0, (int)h->seg1.level_ptr.size(), h->d_plane_lv1, h->g.ny + 1,
                                          h->stream));
        h->rot_device = false;   // the blades now follow the host's list
        // a split step needs every blade stencil cell inside the zone
        if (h->zone_gen == h->marker_gen) h->zone_ok = blades_in_zone(h);
    });
}

// The device's address of p[0, bytes) where a kernel may store there: both ends lie
// in one piece of its own, pinned or managed memory, and the address is aligned.
// NULL where only a copy can go.
static void* device_address(const tdlb_lattice* h, void* p, size_t bytes, size_t align) {
    if ((uintptr_t)p % align) return nullptr;
    char* at[2];
    for (int end = 0; end < 2; end++) {
        cudaPointerAttributes a{};
        if (cudaPointerGetAttributes(&a, (char*)p + (end ? bytes - 1 : 0)) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        const bool writes = a.type == cudaMemoryTypeHost ||
                            ((a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged) && a.device == h->device);
        if (!writes || !a.devicePointer) return nullptr;
        at[end] = (char*)a.devicePointer;
    }
    return at[1] - at[0] == (ptrdiff_t)bytes - 1 ? at[0] : nullptr;
}

// Queue the impeller load of the last forcing pass and its copy into out5.
void queue_impeller_load(tdlb_lattice* h, double* out5) {
    if (!out5) throw Fail{TDLB_EINVAL, "out is NULL"};
    if (h->impeller_begin < 0) throw Fail{TDLB_ESTATE, "no impeller attached (tdlb_attach_rushton)"};
    if (h->pass == 0) throw Fail{TDLB_ESTATE, "no forcing pass yet"};
    tdlb::IbmArgs a = ibm_args(h, 0.f, h->last_beta);
    double* out = h->d_load + tdlb::kLoadBlocks * 5;
    // memory the device can write (its own, pinned host, managed) takes the sums
    // from the kernel; a copy behind it costs 6 us of a small tank's step
    double* direct = (double*)device_address(h, out5, 5 * sizeof(double), alignof(double));
    TDLB_CK(tdlb::launch_marker_load(a, h->d_imp_slots, h->n_imp, h->rot_ci, h->rot_ck, h->d_load, (unsigned*)(out + 5),
                                     direct ? direct : out, h->stream));
    if (!direct) TDLB_CK(cudaMemcpyAsync(out5, out, 5 * sizeof(double), cudaMemcpyDefault, h->stream));
}

int tdlb_impeller_load(tdlb_handle h, double* out5) {
    return guarded<false>(h, [&] {
        queue_impeller_load(h, out5);
        TDLB_CK(cudaStreamSynchronize(h->stream));
    });
}

int tdlb_impeller_load_async(tdlb_handle h, double* out5) {
    return guarded<false>(h, [&] { queue_impeller_load(h, out5); });
}

int tdlb_read_markers(tdlb_handle h, tdlb_marker* out, size_t cap, size_t* n) {
    return guarded(h, [&] {
        if (n) *n = (size_t)h->n_markers;
        if (!out) return;
        if (cap < (size_t)h->n_markers) throw Fail{TDLB_EINVAL, "cap smaller than the marker count"};
        if (h->n_markers)
            TDLB_CK(cudaMemcpyAsync(out, h->d_markers, (size_t)h->n_markers * sizeof(tdlb_marker), cudaMemcpyDeviceToHost,
                                    h->stream));
        TDLB_CK(cudaStreamSynchronize(h->stream));
    });
}

int tdlb_schedule_levels(const tdlb_marker* markers, size_t n, int64_t x, int64_t y, int64_t z, int32_t* level_out,
                         int32_t* max_levels_per_plane) {
    if ((n && !markers) || x < 1 || y < 1 || z < 1 || n > (size_t)0x7fffffff) return TDLB_EINVAL;
    for (size_t q = 0; q < n; q++)
        if (markers[q].i < 0 || markers[q].i >= x || markers[q].j < 0 || markers[q].j >= y || markers[q].k < 0 ||
            markers[q].k >= z)
            return TDLB_EINVAL;
    tdlb::MarkerSchedule s;
    s.build(reinterpret_cast<const tdlb::Marker*>(markers), 0, (int)n, (int)x, (int)y, (int)z, 0, 0);
    if (level_out) {
        // level within its plane, from the plane's first level
        for (int64_t j = 0; j < y; j++)
            for (int lv = s.plane_lv[(size_t)j]; lv < s.plane_lv[(size_t)j + 1]; lv++)
                for (int p = s.level_ptr[(size_t)lv]; p < s.level_ptr[(size_t)lv + 1]; p++)
                    level_out[s.order[(size_t)p]] = lv - s.plane_lv[(size_t)j];
    }
    if (max_levels_per_plane) *max_levels_per_plane = s.max_levels_per_plane;
    return TDLB_OK;
}

int tdlb_debug_set_state(tdlb_handle h, const float* in, int holds_moments) {
    return guarded(h, [&] {
        if (!in) throw Fail{TDLB_EINVAL, "in is NULL"};
        if (h->cfg.storage != TDLB_STORAGE_FP32) throw Fail{TDLB_EINVAL, "raw state access needs FP32 storage"};
        host_aos_to_planes(h, in, tdlb::NQ, h->state_buf());
        h->holds_moments = holds_moments != 0;
        h->initialised = true;
    });
}

int tdlb_debug_transport(tdlb_handle h) {
    return guarded(h, [&] {
        require_init(h);
        if (h->cfg.storage != TDLB_STORAGE_FP32) throw Fail{TDLB_EINVAL, "transport-only steps need FP32 storage"};
        run_step(h, false);
    });
}

}  // extern "C"

namespace tdlb_rt {
void drop_residual_box(tdlb_lattice* h) { ::drop_rbox(h); }
void clear_residual_box(tdlb_lattice* h) { ::clear_rbox(h); }
tdlb::StepArgs step_args(tdlb_lattice* h, bool collide) { return ::step_args(h, collide); }
tdlb::IbmArgs ibm_args(tdlb_lattice* h, float alpha, float beta) { return ::ibm_args(h, alpha, beta); }
void note_pass(tdlb_lattice* h, float beta) {
    h->last_beta = beta;
    h->forced = true;
    h->force_gen = h->marker_gen;
    if (h->list_passes < kSettledPasses) h->list_passes++;
    // blades that turn on the device stay inside the zone's annuli
    h->force_blades_in = h->n_markers == h->n0 || h->rot_device ||
                         (h->zone_gen == h->marker_gen && h->zone_ok);
}
void borrow_stream(tdlb_lattice* h, cudaStream_t s) {
    fence(h);
    cudaStreamSynchronize(h->stream);
    if (!h->own_stream) h->own_stream = h->stream;
    h->stream = s;
}

void return_stream(tdlb_lattice* h) {
    if (!h->own_stream) return;
    h->stream = h->own_stream;
    h->own_stream = nullptr;
    reserve_zone(h);
}

cudaError_t scratch(tdlb_lattice* h, size_t bytes, char** out) {
    if (bytes > h->scratch_bytes) {
        cudaError_t e = cudaStreamSynchronize(h->stream);   // (calls wait for their copies, so nothing uses it)
        if (e != cudaSuccess) return e;
        cudaFree(h->d_scratch);
        h->d_scratch = nullptr;
        h->scratch_bytes = 0;
        e = cudaMalloc(&h->d_scratch, bytes);
        if (e != cudaSuccess) return e;
        h->scratch_bytes = bytes;
    }
    *out = (char*)h->d_scratch;
    return cudaSuccess;
}

void reserve_zone(tdlb_lattice* h) {
    if (h->zone_block || !h->resident || h->own_stream || !(split_wanted(h) || h->rbox_geom.n > 0)) return;
    const size_t nw = (size_t)(h->g.rows() * h->g.jw), ring = (size_t)h->g.ny * sizeof(double2);
    if (cudaMalloc(&h->zone_block, ring + nw * (2 * sizeof(int) + 1)) != cudaSuccess) {
        h->zone_block = nullptr;
        cudaGetLastError();
        return;
    }
    h->d_zone_ring = (double2*)h->zone_block;
    h->d_zone_core = (uint32_t*)(h->zone_block + ring);
    h->d_zone_words = (int*)(h->d_zone_core + nw);
    h->d_zone_skip = (uint8_t*)(h->d_zone_words + nw);
}

void drop_zone(tdlb_lattice* h) {
    cudaFree(h->zone_block);
    h->zone_block = nullptr;
    h->zone_gen = ~0u;
    h->h_zone_core.clear();
}
}  // namespace tdlb_rt
