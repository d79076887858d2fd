// What the launches of the CPU tests' CUDA runtime (fake_cuda.cpp) are held
// against: the buffers that the marker scheduler's and the forcing pass's
// arguments name. k_sched_cells counts the planes' stencil cells and k_zone_core
// marks the blades' annuli, so that the host goes on as with a GPU.
#include <algorithm>
#include <cmath>
#include <set>
#include <string>
#include <vector>

#include "step_kernels.cuh"

void fake_need(const char* who, const char* what, const void* p, long long n);
void fake_fault(const char* who, const char* what);
bool fake_sound();
bool fake_writable(const void* p, long long n);   // pinned or device memory

extern "C" void fake_check(const char* w, void** args) {
    using namespace tdlb;
    const std::string name = w;
    if (name.find("k_sched_") != std::string::npos) {
        const SchedArgs& a = *(const SchedArgs*)args[0];
        fake_need(w, "markers", a.markers, (long long)a.n * sizeof(Marker));
        fake_need(w, "hist", a.hist, (long long)sched_hist_ints(a.g, a.n) * 4);
        fake_need(w, "by_plane", a.by_plane, 4LL * a.n0);
        fake_need(w, "plane_count", a.plane_count, 4LL * a.g.ny);
        if (name.find("k_sched_cells") != std::string::npos && fake_sound()) {
            std::vector<std::set<long long>> cells((size_t)a.g.ny);
            for (int q = 0; q < a.n0; q++) {
                const Marker& m = a.markers[q];
                if (m.i < 0 || m.i >= a.g.nx || m.j < 0 || m.j >= a.g.ny || m.k < 0 || m.k >= a.g.nz) {
                    a.info[0] = std::min(a.info[0], q);
                    continue;
                }
                for (int di = -1; di <= 1; di++)
                    for (int dk = -1; dk <= 1; dk++)
                        cells[(size_t)m.j].insert((m.i + di + a.g.nx) % a.g.nx * a.g.nz + (m.k + dk + a.g.nz) % a.g.nz);
            }
            for (int j = 0; j < a.g.ny; j++) a.plane_count[j] = (int)cells[(size_t)j].size();
        }
        if (name.find("k_sched_levels") != std::string::npos) {
            long long cells = 0;
            for (int j = 0; j < a.g.ny; j++) cells += a.plane_count[j];
            fake_need(w, "owner", a.owner, 4 * cells);
            fake_need(w, "cell_e", a.cell_e, 4 * cells);
            fake_need(w, "sched", a.sched, 4LL * a.n0);
            fake_need(w, "prep", a.prep, 4LL * PF_STRIDE * a.n0);
            fake_need(w, "level_ptr", a.level_ptr, 4LL * (a.n0 + 1));
            fake_need(w, "plane_lv0", a.plane_lv0, 4LL * (a.g.ny + 1));
            fake_need(w, "plane_lv1", a.plane_lv1, 4LL * (a.g.ny + 1));
            fake_need(w, "mask_static", a.mask_static, 4 * a.g.rows() * a.g.jw);
        }
    }
    if (name.find("k_zone_core") != std::string::npos && *(const double2* const*)args[2]) {
        const Dims& g = *(const Dims*)args[0];
        const double2* ring = *(const double2* const*)args[2];
        const double ci = *(const double*)args[3], ck = *(const double*)args[4];
        uint32_t* core = *(uint32_t* const*)args[5];
        fake_need(w, "core", core, 4 * g.rows() * g.jw);
        fake_need(w, "ring", ring, 16LL * g.ny);
        for (int i = 0; i < g.nx && fake_sound(); i++)
            for (int k = 0; k < g.nz; k++)
                for (int j = 0; j < g.ny; j++) {
                    const double d = std::sqrt((i - ci) * (i - ci) + (k - ck) * (k - ck));
                    if (ring[j].y >= 0.0 && d >= ring[j].x && d <= ring[j].y) core[g.word(i, j, k)] |= 1u << (j & 31);
                }
    }
    if (name.find("k_marker_load(") != std::string::npos) {
        const double* out = *(double* const*)args[7];
        if ((uintptr_t)out % 8) fake_fault(w, "the load's address is not a multiple of 8");
        if (!fake_writable(out, 40)) fake_fault(w, "the load does not lie in memory that the device can write");
    }
    if (name.find("k_rotate_markers") != std::string::npos) {
        const int n = *(const int*)args[2];
        fake_need(w, "offsets", *(const double* const*)args[0], 16LL * n);
        fake_need(w, "markers", *(Marker* const*)args[1], (long long)n * sizeof(Marker));
    }
    if (name.find("k_ibm_gather<") != std::string::npos || name.find("k_ibm_spread<") != std::string::npos) {
        const IbmArgs& a = *(const IbmArgs*)args[0];
        fake_need(w, "markers", a.markers, (long long)a.n * sizeof(Marker));
        fake_need(w, "sched", a.sched, 4LL * a.n);
        fake_need(w, "sums", a.sums, 12LL * a.n);
        fake_need(w, "cell_e", a.cell_e, 4LL * (a.ncell + 16));
        fake_need(w, "cell_m", a.cell_m, 16LL * a.ncell + 64);
        fake_need(w, "cell_F", a.cell_F, 12LL * a.ncell + 64);
        fake_need(w, "prep", a.prep, 4LL * PF_STRIDE * a.n0);
        fake_need(w, "tail", a.tail, a.n > a.n0 ? 4LL * TF_COUNT * a.tail_cap : 0);
        if (a.n - a.n0 > a.tail_cap) fake_fault(w, "tail is shorter than the blades");
        fake_need(w, "plane_lv1", a.plane_lv1, 4LL * (a.g.ny + 1));
        fake_need(w, "plane_cell", a.plane_cell, 4LL * (a.g.ny + 1));
        fake_need(w, "plane_list", a.plane_list, 4LL * a.g.ny);
    }
}

// index arithmetic that kernels and launches share
extern "C" long long fake_listed_word(unsigned block, unsigned thread, unsigned V) { return tdlb::listed_word(block, thread, V); }
extern "C" long long fake_listed_blocks(long long words, unsigned V) { return tdlb::listed_blocks(words, V); }
extern "C" void fake_gather_item(int tank, int j0, int p0, int* out4) {
    const tdlb::GatherItem g = tdlb::GatherItem::of(tdlb::GatherItem::cells(tank, j0, p0));
    out4[0] = g.tank;
    out4[1] = g.kind;
    out4[2] = g.j0();
    out4[3] = g.p0();
}
extern "C" void fake_pull_span(int nx, int ny, int nz, int d, int es, int eso, int even, long long e0, long long e1, long long* out2) {
    const tdlb::PrefetchSpan s = tdlb::pull_span(tdlb::make_dims(nx, ny, nz), d, es, eso != 0, even != 0, e0, e1);
    out2[0] = s.lo;
    out2[1] = s.hi;
}
extern "C" int fake_prefetch_tiles() { return tdlb::kPrefetchTiles; }
extern "C" int fake_row_pitch(int nx, int ny, int nz) { return tdlb::make_dims(nx, ny, nz).jp; }
