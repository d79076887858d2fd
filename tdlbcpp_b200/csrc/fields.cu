// Field read-back: the interior cells' moments, density, velocity, force, eddy
// viscosity and touched flags in the reference's cell order (i, j, k), k
// fastest, into the caller's memory.
//
// One kernel per field computes the values where the lattice lies and turns
// them round (rows run along j) through shared memory, for a slab of i at a
// time; the slab's rows then go to the caller in one copy per output. The
// first form copied all 18 moment planes of the padded lattice to the host and
// picked the values there, one thread: 240 ms for the fields of a 128^3
// tank, of which 67 MB are the result.
#include "tdlb_handle.hpp"
#include "step_kernels.cuh"

#include <sys/mman.h>
#include <unistd.h>
#ifndef MADV_POPULATE_WRITE   // Linux 5.14
#define MADV_POPULATE_WRITE 23
#endif

#include <algorithm>
#include <atomic>
#include <string>
#include <thread>
#include <vector>

namespace tdlb {

// What a cell's outputs are made of.
struct FieldArgs {
    Planes A;
    Dims g;
    int mode, even;
    CollideParams p;
    ResidualBox rb;
    const float4* F;
    const uint32_t* mask;
    const float* Nu;
};
__device__ __forceinline__ float4 field_force(const FieldArgs& a, int i, int j, int k) {
    const bool on = (a.mask[a.g.word(i, j, k)] >> (j & 31)) & 1u;
    return on ? a.F[a.g.at(i, j, k)] : make_float4(0.f, 0.f, 0.f, 0.f);
}

// The values of one cell. N per cell; the first `split` go to the first
// output array, the rest to the second.
template <typename S>
struct MomentsOf {
    static constexpr int N = NQ, SPLIT = NQ;
    __device__ static void get(const FieldArgs& a, int i, int j, int k, float (&v)[N]) {
        state_moments18<S>(a.A, a.g, a.mode, a.even, a.p, i, j, k, v, a.rb);
    }
};
// density and u = (1 / rho) (j + F / 2) (QVec.hpp:385-394, in its precision)
template <typename S>
struct VelocityOf {
    static constexpr int N = 4, SPLIT = 1;
    __device__ static void get(const FieldArgs& a, int i, int j, int k, float (&v)[N]) {
        float m[NQ];
        state_moments18<S>(a.A, a.g, a.mode, a.even, a.p, i, j, k, m, a.rb);
        const float4 f = field_force(a, i, j, k);
        const double r = __ddiv_rn(1.0, (double)m[0]);
        v[0] = m[0];
        v[1] = (float)__dmul_rn(r, __dadd_rn((double)m[1], 0.5 * (double)f.x));
        v[2] = (float)__dmul_rn(r, __dadd_rn((double)m[2], 0.5 * (double)f.y));
        v[3] = (float)__dmul_rn(r, __dadd_rn((double)m[3], 0.5 * (double)f.z));
    }
};
struct ForceOf {
    static constexpr int N = 3, SPLIT = 3;
    __device__ static void get(const FieldArgs& a, int i, int j, int k, float (&v)[N]) {
        const float4 f = field_force(a, i, j, k);
        v[0] = f.x;
        v[1] = f.y;
        v[2] = f.z;
    }
};
struct NuOf {
    static constexpr int N = 1, SPLIT = 1;
    __device__ static void get(const FieldArgs& a, int i, int j, int k, float (&v)[N]) { v[0] = a.Nu[a.g.at(i, j, k)]; }
};
struct StateOf {   // the 18 raw values at the cell's element (FP32 storage)
    static constexpr int N = NQ, SPLIT = NQ;
    __device__ static void get(const FieldArgs& a, int i, int j, int k, float (&v)[N]) {
#pragma unroll
        for (int d = 0; d < NQ; d++) v[d] = a.A.p[d][a.g.at(i, j, k)];
    }
};

// Tile of 32 cells along j and KT along k of one i: lanes run along j while the
// values are made (coalesced on the lattice), then along the output row of
// each j, KT cells of N values (contiguous there). out1: values [0, SPLIT) of
// the slab's cells; out2: the rest, interleaved per cell, or (stride2 > 0) each in
// an array of its own, stride2 apart.
template <typename FIELD, int KT>
__global__ void __launch_bounds__(256) k_fields(FieldArgs a, int i0, float* __restrict__ out1, float* __restrict__ out2,
                                                long long stride2) {
    constexpr int N = FIELD::N, SPLIT = FIELD::SPLIT, REST = N - SPLIT, ROW = KT * N + 1;   // odd: no bank conflicts
    static_assert(KT % 8 == 0, "eight warps along k");
    __shared__ float tile[32 * ROW];
    const Dims& g = a.g;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = i0 + (int)blockIdx.z, j0 = (int)blockIdx.x * 32, k0 = (int)blockIdx.y * KT;
    const int j = j0 + lane;
#pragma unroll
    for (int q = 0; q < KT / 8; q++) {
        const int kk = warp + 8 * q, k = k0 + kk;
        if (j < g.ny && k < g.nz) {
            float v[N];
            FIELD::get(a, i, j, k, v);
#pragma unroll
            for (int c = 0; c < N; c++) tile[lane * ROW + kk * N + c] = v[c];
        }
    }
    __syncthreads();
    const int nk = min(KT, g.nz - k0);
    for (int jj = warp; jj < 32 && j0 + jj < g.ny; jj += 8) {
        const long long cell = ((long long)blockIdx.z * g.ny + (j0 + jj)) * g.nz + k0;
        const float* t = tile + jj * ROW;
        for (int x = lane; x < nk * SPLIT; x += 32) out1[cell * SPLIT + x] = t[x / SPLIT * N + x % SPLIT];
        if constexpr (REST > 0) {
            if (stride2 == 0) {
                for (int x = lane; x < nk * REST; x += 32) out2[cell * REST + x] = t[x / REST * N + SPLIT + x % REST];
            } else {
                for (int c = 0; c < REST; c++)
                    for (int x = lane; x < nk; x += 32) out2[c * stride2 + cell + x] = t[x * N + SPLIT + c];
            }
        }
    }
}

// Touched flags, a byte per cell.
__global__ void __launch_bounds__(256) k_touched(const uint32_t* __restrict__ mask, Dims g, int i0, long long n,
                                                 uint8_t* __restrict__ out) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int k = (int)(t % g.nz);
    const long long l = t / g.nz;
    const int j = (int)(l % g.ny), i = i0 + (int)(l / g.ny);
    out[t] = (uint8_t)((mask[g.word(i, j, k)] >> (j & 31)) & 1u);
}

}  // namespace tdlb

namespace {

struct FFail {
    int code;
    std::string msg;
};

#define TDLB_FCK(call)                                                                                      \
    do {                                                                                                    \
        cudaError_t e_ = (call);                                                                            \
        if (e_ != cudaSuccess) throw FFail{TDLB_ECUDA, tdlb_rt::error_text(#call, e_)};                     \
    } while (0)

template <bool INIT = true, typename F>
int fguard(tdlb_lattice* h, const void* out, F&& fn) {
    if (!h) return TDLB_EINVAL;
    try {
        cudaSetDevice(h->device);
        tdlb_rt::fence(h);
        if (INIT && !h->initialised) throw FFail{TDLB_ESTATE, "call tdlb_initialise() first"};
        if (!out) throw FFail{TDLB_EINVAL, "out is NULL"};
        fn();
        return TDLB_OK;
    } catch (const FFail& f) {
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

// One output array of a read: `per` bytes per cell at `dst` (NULL: not wanted),
// from byte offset `off` per cell of the slab's device scratch.
struct Out {
    void* dst;
    size_t per;
};

// Populates the pages of the caller's buffers from a few threads while the
// device works and the first copies run: a copy into fresh memory (a new numpy
// array) otherwise faults its pages in one by one, 5 GB/s against 20 into
// memory already mapped (64 MB: 13.4 against 3.3 ms). The contents are left
// alone, and nothing depends on it: kernels without MADV_POPULATE_WRITE, or a
// buffer that cannot be populated, only copy more slowly.
class Populate {
public:
    // ranges in the order the copies will take them
    explicit Populate(const std::vector<std::pair<char*, size_t>>& ranges) {
        size_t total = 0;
        for (const auto& r : ranges) total += r.second;
        if (total < kLeast) return;
        // whole huge pages where the caller's memory has them
        for (const auto& r : ranges) {
            const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
            const uintptr_t hi = ((uintptr_t)r.first + r.second) / page * page;
            for (uintptr_t a = ((uintptr_t)r.first + page - 1) / page * page; a < hi;) {
                const uintptr_t e = std::min(hi, (a / kPiece + 1) * kPiece);
                pieces_.emplace_back(a, e - a);
                a = e;
            }
        }
        const unsigned hw = std::thread::hardware_concurrency();
        const size_t n = std::min<size_t>(std::max(1u, std::min(8u, hw / 2)), total / kLeast + 1);
        try {
            for (size_t t = 0; t < n; t++)
                threads_.emplace_back([this] {
                    for (size_t q; (q = next_.fetch_add(1)) < pieces_.size();)
                        if (madvise((void*)pieces_[q].first, pieces_[q].second, MADV_POPULATE_WRITE) != 0) return;
                });
        } catch (const std::exception&) {
            // no more threads: the copies do without
        }
    }
    Populate(const Populate&) = delete;
    Populate& operator=(const Populate&) = delete;
    ~Populate() {
        for (std::thread& t : threads_) t.join();
    }

private:
    static constexpr size_t kLeast = (size_t)4 << 20, kPiece = (size_t)4 << 20;
    std::vector<std::pair<uintptr_t, size_t>> pieces_;
    std::atomic<size_t> next_{0};
    std::vector<std::thread> threads_;
};

char* scratch(tdlb_lattice* h, size_t bytes) {
    char* p = nullptr;
    TDLB_FCK(tdlb_rt::scratch(h, bytes, &p));
    return p;
}

// Slabs of i of at most about this many bytes of output at a time: enough for
// full copy rate, and all the memory a read of any size needs.
constexpr size_t kSlabBytes = (size_t)32 << 20;

// For every slab: launch(i0, ni, base) fills the slab's outputs one after
// another from `base` (each starting on a 256-byte boundary), which then go
// to the caller.
template <typename L>
void read_out(tdlb_lattice* h, const std::vector<Out>& outs, L&& launch) {
    const Dims& g = h->g;
    const size_t line = (size_t)g.ny * g.nz;
    size_t per = 0;
    for (const Out& o : outs) per += o.per;
    const int ni = (int)std::min<size_t>((size_t)g.nx, std::max<size_t>(1, kSlabBytes / (per * line)));
    std::vector<size_t> at(outs.size());
    size_t bytes = 0;
    for (size_t q = 0; q < outs.size(); q++) {
        at[q] = bytes;
        bytes += (outs[q].per * line * (size_t)ni + 255) / 256 * 256;
    }
    char* base = scratch(h, bytes);
    std::vector<std::pair<char*, size_t>> ranges;
    for (int i0 = 0; i0 < g.nx; i0 += ni)
        for (const Out& o : outs)
            if (o.dst) ranges.emplace_back((char*)o.dst + o.per * line * (size_t)i0, o.per * line * (size_t)std::min(ni, g.nx - i0));
    Populate populate(ranges);
    for (int i0 = 0; i0 < g.nx; i0 += ni) {
        const int n = std::min(ni, g.nx - i0);
        launch(i0, n, base, at);
        TDLB_FCK(cudaGetLastError());
        for (size_t q = 0; q < outs.size(); q++)
            if (outs[q].dst)
                TDLB_FCK(cudaMemcpyAsync((char*)outs[q].dst + outs[q].per * line * (size_t)i0, base + at[q],
                                         outs[q].per * line * (size_t)n, cudaMemcpyDeviceToHost, h->stream));
    }
    TDLB_FCK(cudaStreamSynchronize(h->stream));
}

tdlb::FieldArgs field_args(tdlb_lattice* h) {
    tdlb::FieldArgs a{};
    a.A = h->planes(h->state_buf());
    a.g = h->g;
    a.mode = h->state_mode();
    a.even = h->even ? 1 : 0;
    a.p = h->cp;
    a.rb = h->rbox(h->state_index());
    a.F = reinterpret_cast<const float4*>(h->F);
    a.mask = h->mask_cur();
    a.Nu = h->Nu;
    return a;
}

template <typename FIELD, int KT>
void launch_fields(const tdlb_lattice* h, const tdlb::FieldArgs& a, int i0, int n, float* out1, float* out2,
                   long long stride2) {
    const Dims& g = a.g;
    const dim3 grid((unsigned)((g.ny + 31) / 32), (unsigned)((g.nz + KT - 1) / KT), (unsigned)n);
    tdlb::k_fields<FIELD, KT><<<grid, 256, 0, h->stream>>>(a, i0, out1, out2, stride2);
}

// Density and velocity: rho and either three arrays or (u3) one interleaved.
void read_velocity(tdlb_lattice* h, float* rho, float* const (&u)[3], float* u3) {
    const tdlb::FieldArgs a = field_args(h);
    std::vector<Out> outs = {{rho, 4}};
    if (u3) outs.push_back({u3, 12});
    else for (float* c : u) outs.push_back({c, 4});
    read_out(h, outs, [&](int i0, int n, char* base, const std::vector<size_t>& at) {
        const long long stride = u3 ? 0 : (long long)(at[2] - at[1]) / 4;
        tdlb::with_storage(h->cfg.storage, [&](auto s) {
            launch_fields<tdlb::VelocityOf<decltype(s)>, 32>(h, a, i0, n, (float*)(base + at[0]), (float*)(base + at[1]), stride);
        });
    });
}

template <typename FIELD, int KT>
void read_one(tdlb_lattice* h, float* out) {
    const tdlb::FieldArgs a = field_args(h);
    read_out(h, {{out, FIELD::N * sizeof(float)}}, [&](int i0, int n, char* base, const std::vector<size_t>& at) {
        launch_fields<FIELD, KT>(h, a, i0, n, (float*)(base + at[0]), nullptr, 0);
    });
}

}  // namespace

extern "C" {

int tdlb_read_moments(tdlb_handle h, float* out) {
    return fguard(h, out, [&] {
        tdlb::with_storage(h->cfg.storage, [&](auto s) { read_one<tdlb::MomentsOf<decltype(s)>, 8>(h, out); });
    });
}

int tdlb_read_velocity_density(tdlb_handle h, float* rho, float* ux, float* uy, float* uz) {
    return fguard(h, h, [&] {
        if (!rho && !ux && !uy && !uz) return;
        read_velocity(h, rho, {ux, uy, uz}, nullptr);
    });
}

int tdlb_read_density_velocity3(tdlb_handle h, float* rho, float* u3) {
    return fguard(h, u3, [&] { read_velocity(h, rho, {nullptr, nullptr, nullptr}, u3); });
}

int tdlb_read_force(tdlb_handle h, float* f3) {
    return fguard(h, f3, [&] { read_one<tdlb::ForceOf, 32>(h, f3); });
}

int tdlb_read_nu(tdlb_handle h, float* nu) {
    return fguard(h, nu, [&] { read_one<tdlb::NuOf, 32>(h, nu); });
}

int tdlb_read_touched(tdlb_handle h, uint8_t* flags) {
    return fguard(h, flags, [&] {
        const uint32_t* mask = h->mask_cur();
        read_out(h, {{flags, 1}}, [&](int i0, int n, char* base, const std::vector<size_t>& at) {
            const long long cells = (long long)n * h->g.ny * h->g.nz;
            tdlb::k_touched<<<(unsigned)((cells + 255) / 256), 256, 0, h->stream>>>(mask, h->g, i0, cells,
                                                                                   (uint8_t*)(base + at[0]));
        });
    });
}

int tdlb_debug_get_state(tdlb_handle h, float* out) {
    return fguard<false>(h, out, [&] {
        if (h->cfg.storage != TDLB_STORAGE_FP32) throw FFail{TDLB_EINVAL, "raw state access needs FP32 storage"};
        read_one<tdlb::StateOf, 8>(h, out);
    });
}

}  // extern "C"
