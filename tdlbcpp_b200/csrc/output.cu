// Output kernels: vorticity slices and the XZ plane dump, with the
// reference's excluded output points.
//
//   vorticity  calcVorticityXZ / calcVorticityXY (ComputeUnitOutput.hpp:113-285,
//              GPU ComputeUnitOutput.cuh:10-64): log |curl u|^2 from central
//              differences of u = j / rho (QVec::velocity(), QVec.hpp:136-144)
//              of the moments the reference's Q holds between steps;
//              excluded cells give -1 (the GPU kernel's value).
//   plane      savePlaneXZ<float, 4> (ComputeUnitOutput.hpp:354-447): for
//              every non-excluded cell of the plane, in (i, k) order, a
//              tDiskGrid<float, 4> record (Output.hpp:22-26) of Q slots 0..3
//              (Simple: the first four moments; Esotwist: the raw slots,
//              see k_plane_xz), and a tDiskGrid<float, 3> record of F where
//              F is non-zero.
//   exclude    setOutputExcludePoints / unsetOutputExcludePoints
//              (ComputeUnitOutput.hpp:20-53): one bit per cell.
//
// Neighbours beyond the lattice faces: the reference reads its ghost layer
// there, which its step never fills with moments (Simple: the streamed-out
// populations of the bounce-back; Esotwist: the initial values), so those
// cells' vorticity is not meaningful in the reference. Here the cell itself
// stands in for the missing neighbour.
#include "tdlb_handle.hpp"
#include "step_kernels.cuh"

#include <algorithm>
#include <string>
#include <vector>

namespace tdlb {

// u = j / rho of cell (i, j, k), clamped into the lattice.
template <typename S>
__device__ __forceinline__ void cell_velocity(const Planes& A, const Dims& g, int mode, int even, const CollideParams& p,
                                              int i, int j, int k, float (&u)[3]) {
    i = min(max(i, 0), g.nx - 1);
    j = min(max(j, 0), g.ny - 1);
    k = min(max(k, 0), g.nz - 1);
    float m[NQ];
    state_moments18<S>(A, g, mode, even, p, i, j, k, m);
    u[0] = m[1] / m[0];
    u[1] = m[2] / m[0];
    u[2] = m[3] / m[0];
}

// axis 1: XZ slice at j = cut, out[i * z + k]; axis 2: XY slice at k = cut,
// out[j * x + i] (the reference's picture layouts).
template <typename S>
__global__ void __launch_bounds__(256) k_vorticity(Planes A, Dims g, int mode, int even, CollideParams p, int axis,
                                                   int cut, const uint32_t* __restrict__ excl, float* __restrict__ out) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int i, j, k;
    long long o;
    if (axis == 1) {
        if (t >= (long long)g.nx * g.nz) return;
        i = (int)(t / g.nz);
        k = (int)(t - (long long)i * g.nz);
        j = cut;
        o = (long long)i * g.nz + k;
    } else {
        if (t >= (long long)g.nx * g.ny) return;
        j = (int)(t / g.nx);
        i = (int)(t - (long long)j * g.nx);
        k = cut;
        o = (long long)j * g.nx + i;
    }
    if (excl && ((excl[g.word(i, j, k)] >> (j & 31)) & 1u)) {
        out[o] = -1.f;
        return;
    }
    float q05[3], q06[3], q03[3], q04[3], q01[3], q02[3];
    cell_velocity<S>(A, g, mode, even, p, i, j, k + 1, q05);
    cell_velocity<S>(A, g, mode, even, p, i, j, k - 1, q06);
    cell_velocity<S>(A, g, mode, even, p, i, j + 1, k, q03);
    cell_velocity<S>(A, g, mode, even, p, i, j - 1, k, q04);
    cell_velocity<S>(A, g, mode, even, p, i + 1, j, k, q01);
    cell_velocity<S>(A, g, mode, even, p, i - 1, j, k, q02);
    const float uxy = 0.5f * (q05[0] - q06[0]);
    const float uxz = 0.5f * (q03[0] - q04[0]);
    const float uyx = 0.5f * (q01[1] - q02[1]);
    const float uyz = 0.5f * (q03[1] - q04[1]);
    const float uzx = 0.5f * (q01[2] - q02[2]);
    const float uzy = 0.5f * (q05[2] - q06[2]);
    const float a = uxy - uyx, b = uyz - uzy, c = uzx - uxz;
    out[o] = logf(b * b + c * c + a * a);
}

// The XZ plane dump: the record of every cell that is not excluded, in (i, k)
// order, and of every such cell whose F is not zero, packed on the device
// (counts per block, their running sums, the records), so that only the records
// cross to the host. (It was 32 bytes of every cell, a fresh device buffer per
// call and a host pass over them, twice where a caller asks for the counts
// first.)
struct PlaneArgs {
    Dims g;
    int j;
    const float4* F;
    const uint32_t* mask;
    const uint32_t* excl;
    int2* offset;                 // [blocks + 1] records before each block; the totals
    tdlb_disk_grid4* q;
    tdlb_disk_grid3* f;
};
// the cell of a thread; its F (zero where the last pass did not touch it)
__device__ __forceinline__ bool plane_cell(const PlaneArgs& a, int& i, int& k, float4& v) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    i = (int)(t / a.g.nz);
    k = (int)(t - (long long)i * a.g.nz);
    v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t >= a.g.rows()) return false;
    const long long w = a.g.word(i, a.j, k);
    if (a.excl && ((a.excl[w] >> (a.j & 31)) & 1u)) return false;
    if ((a.mask[w] >> (a.j & 31)) & 1u) v = a.F[a.g.at(i, a.j, k)];
    return true;
}
__device__ __forceinline__ bool not_zero(const float4& v) { return v.x != 0.f || v.y != 0.f || v.z != 0.f; }   // Force::isNotZero

__global__ void __launch_bounds__(256) k_plane_count(PlaneArgs a) {
    int i, k;
    float4 v;
    const bool in = plane_cell(a, i, k, v);
    const int nq = __syncthreads_count(in), nf = __syncthreads_count(in && not_zero(v));
    if (threadIdx.x == 0) a.offset[blockIdx.x] = make_int2(nq, nf);
}

__global__ void __launch_bounds__(32) k_plane_offsets(PlaneArgs a, int blocks) {
    int2 carry = make_int2(0, 0);
    const int lane = threadIdx.x;
    for (int b = 0; b < blocks; b += 32) {
        const int2 x = b + lane < blocks ? a.offset[b + lane] : make_int2(0, 0);
        int2 s = x;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const int p = __shfl_up_sync(0xffffffffu, s.x, d), q = __shfl_up_sync(0xffffffffu, s.y, d);
            if (lane >= d) {
                s.x += p;
                s.y += q;
            }
        }
        if (b + lane < blocks) a.offset[b + lane] = make_int2(carry.x + s.x - x.x, carry.y + s.y - x.y);
        carry.x += __shfl_sync(0xffffffffu, s.x, 31);
        carry.y += __shfl_sync(0xffffffffu, s.y, 31);
    }
    if (lane == 0) a.offset[blocks] = carry;
}

// Q slots 0..3 as the reference holds them. Simple: the cell's own first four
// moments. Esotwist: the reference's savePlaneXZ copies the raw slots of its Q,
// which after moments() hold the writeMoments placement -- slot s at location
// x is moment d = (even ? s : s^1) of cell x - max(-c_d, 0) (wrapping) -- so
// each slot is that moment of that cell.
template <typename S>
__global__ void __launch_bounds__(256) k_plane_xz(PlaneArgs a, Planes A, int mode, int even, CollideParams p, int esotwist) {
    __shared__ int2 warps[8];
    const Dims& g = a.g;
    const int j = a.j, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int i, k;
    float4 v;
    const bool in = plane_cell(a, i, k, v), force = in && not_zero(v);
    const unsigned vq = __ballot_sync(0xffffffffu, in), vf = __ballot_sync(0xffffffffu, force);
    if (lane == 0) warps[warp] = make_int2(__popc(vq), __popc(vf));
    __syncthreads();
    if (!in) return;
    int2 at = a.offset[blockIdx.x];
    for (int w = 0; w < warp; w++) {
        at.x += warps[w].x;
        at.y += warps[w].y;
    }
    at.x += __popc(vq & ((1u << lane) - 1u));
    at.y += __popc(vf & ((1u << lane) - 1u));
    tdlb_disk_grid4 r;
    r.iGrid = (uint16_t)i;
    r.jGrid = (uint16_t)j;        // savePlaneXZ: j - 1 in ghosted cells
    r.kGrid = (uint16_t)k;
    r.pad = 0;
    float m[NQ];
    if (!esotwist) {
        state_moments18<S>(A, g, mode, even, p, i, j, k, m);
#pragma unroll
        for (int s = 0; s < 4; s++) r.q[s] = m[s];
    } else {
#pragma unroll
        for (int s = 0; s < 4; s++) {
            const int d = even ? s : (s ^ 1);
            const int si = cx_of(d) < 0 ? (i == 0 ? g.nx - 1 : i - 1) : i;
            const int sj = cy_of(d) < 0 ? (j == 0 ? g.ny - 1 : j - 1) : j;
            const int sk = cz_of(d) < 0 ? (k == 0 ? g.nz - 1 : k - 1) : k;
            state_moments18<S>(A, g, mode, even, p, si, sj, sk, m);
            r.q[s] = even ? m[s] : m[s ^ 1];
        }
    }
    a.q[at.x] = r;
    if (force) {
        tdlb_disk_grid3 rf;
        rf.iGrid = (uint16_t)i;
        rf.jGrid = (uint16_t)(j + 1);  // savePlaneXZ writes the ghosted j for F
        rf.kGrid = (uint16_t)k;
        rf.pad = 0;
        rf.q[0] = v.x;
        rf.q[1] = v.y;
        rf.q[2] = v.z;
        a.f[at.y] = rf;
    }
}

}  // namespace tdlb

namespace {

struct OFail {
    int code;
    std::string msg;
};

#define TDLB_OCK(call)                                                                                      \
    do {                                                                                                    \
        cudaError_t e_ = (call);                                                                            \
        if (e_ != cudaSuccess) throw OFail{TDLB_ECUDA, tdlb_rt::error_text(#call, e_)};                     \
    } while (0)

template <typename F>
int oguard(tdlb_lattice* h, F&& fn) {
    if (!h) return TDLB_EINVAL;
    try {
        cudaSetDevice(h->device);
        tdlb_rt::fence(h);
        fn();
        return TDLB_OK;
    } catch (const OFail& f) {
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

void require(tdlb_lattice* h) {
    if (!h->initialised) throw OFail{TDLB_ESTATE, "not initialised (tdlb_initialise)"};
}

// The handle's device scratch.
char* scratch(tdlb_lattice* h, size_t bytes) {
    char* p = nullptr;
    TDLB_OCK(tdlb_rt::scratch(h, bytes, &p));
    return p;
}

unsigned blocks(long long n) { return (unsigned)((n + 255) / 256); }

}  // namespace

extern "C" {

int tdlb_set_output_exclude(tdlb_handle h, const tdlb_marker* markers, size_t n, int exclude) {
    return oguard(h, [&] {
        if (n && !markers) throw OFail{TDLB_EINVAL, "markers is NULL"};
        const Dims& g = h->g;
        for (size_t q = 0; q < n; q++)
            if (markers[q].i < 0 || markers[q].i >= g.nx || markers[q].j < 0 || markers[q].j >= g.ny ||
                markers[q].k < 0 || markers[q].k >= g.nz)
                throw OFail{TDLB_EINVAL, "marker " + std::to_string(q) + " outside the interior"};
        if (h->h_exclude.empty()) h->h_exclude.assign((size_t)h->mask_words, 0u);
        for (size_t q = 0; q < n; q++) {
            const int j = (int)markers[q].j;
            uint32_t& w = h->h_exclude[(size_t)g.word((int)markers[q].i, j, (int)markers[q].k)];
            if (exclude) w |= 1u << (j & 31);
            else w &= ~(1u << (j & 31));
        }
        if (!h->d_exclude) TDLB_OCK(cudaMalloc(&h->d_exclude, (size_t)h->mask_words * sizeof(uint32_t)));
        TDLB_OCK(cudaMemcpyAsync(h->d_exclude, h->h_exclude.data(), h->h_exclude.size() * sizeof(uint32_t),
                                 cudaMemcpyHostToDevice, h->stream));
        TDLB_OCK(cudaStreamSynchronize(h->stream));
    });
}

static int vorticity(tdlb_handle h, int axis, int64_t cut, float* out) {
    return oguard(h, [&] {
        require(h);
        const Dims& g = h->g;
        const long long lim = axis == 1 ? g.ny : g.nz;
        if (!out || cut < 0 || cut >= lim) throw OFail{TDLB_EINVAL, "cut outside the lattice or out is NULL"};
        const long long n = axis == 1 ? (long long)g.nx * g.nz : (long long)g.nx * g.ny;
        float* d = (float*)scratch(h, (size_t)n * sizeof(float));
        const Planes A = h->planes(h->state_buf());
        const int mode = h->state_mode(), even = h->even ? 1 : 0;
        tdlb::with_storage(h->cfg.storage, [&](auto s) {
            tdlb::k_vorticity<decltype(s)><<<blocks(n), 256, 0, h->stream>>>(A, g, mode, even, h->cp, axis, (int)cut,
                                                                            h->d_exclude, d);
        });
        TDLB_OCK(cudaGetLastError());
        TDLB_OCK(cudaMemcpyAsync(out, d, (size_t)n * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
        TDLB_OCK(cudaStreamSynchronize(h->stream));
    });
}

int tdlb_vorticity_xz(tdlb_handle h, int64_t j, float* out) { return vorticity(h, 1, j, out); }
int tdlb_vorticity_xy(tdlb_handle h, int64_t k, float* out) { return vorticity(h, 2, k, out); }

int tdlb_plane_xz(tdlb_handle h, int64_t j, tdlb_disk_grid4* q_out, size_t q_cap, size_t* q_n, tdlb_disk_grid3* f_out,
                  size_t f_cap, size_t* f_n) {
    return oguard(h, [&] {
        require(h);
        const Dims& g = h->g;
        if (j < 0 || j >= g.ny) throw OFail{TDLB_EINVAL, "j outside the lattice"};
        if (!q_n || !f_n) throw OFail{TDLB_EINVAL, "q_n and f_n are required"};
        const long long n = g.rows();
        const int nb = (int)blocks(n);
        auto up = [](size_t b) { return (b + 255) / 256 * 256; };
        const size_t b_off = up((size_t)(nb + 1) * sizeof(int2)), b_q = up((size_t)n * sizeof(tdlb_disk_grid4));
        const size_t b_f = up((size_t)n * sizeof(tdlb_disk_grid3));
        char* base = scratch(h, b_off + (q_out || f_out ? b_q + b_f : 0));
        tdlb::PlaneArgs a{g, (int)j, reinterpret_cast<const float4*>(h->F), h->mask_cur(), h->d_exclude, (int2*)base,
                          (tdlb_disk_grid4*)(base + b_off), (tdlb_disk_grid3*)(base + b_off + b_q)};
        tdlb::k_plane_count<<<nb, 256, 0, h->stream>>>(a);
        tdlb::k_plane_offsets<<<1, 32, 0, h->stream>>>(a, nb);
        if (q_out || f_out) {
            const Planes A = h->planes(h->state_buf());
            const int mode = h->state_mode(), even = h->even ? 1 : 0;
            tdlb::with_storage(h->cfg.storage, [&](auto s) {
                tdlb::k_plane_xz<decltype(s)><<<nb, 256, 0, h->stream>>>(a, A, mode, even, h->cp,
                                                                       h->cfg.streaming == TDLB_STREAMING_ESOTWIST);
            });
        }
        TDLB_OCK(cudaGetLastError());
        int2 total;
        TDLB_OCK(cudaMemcpyAsync(&total, a.offset + nb, sizeof total, cudaMemcpyDeviceToHost, h->stream));
        TDLB_OCK(cudaStreamSynchronize(h->stream));
        const size_t nq = (size_t)total.x, nf = (size_t)total.y;
        if (q_out && std::min(nq, q_cap))
            TDLB_OCK(cudaMemcpyAsync(q_out, a.q, std::min(nq, q_cap) * sizeof *q_out, cudaMemcpyDeviceToHost, h->stream));
        if (f_out && std::min(nf, f_cap))
            TDLB_OCK(cudaMemcpyAsync(f_out, a.f, std::min(nf, f_cap) * sizeof *f_out, cudaMemcpyDeviceToHost, h->stream));
        TDLB_OCK(cudaStreamSynchronize(h->stream));
        *q_n = nq;
        *f_n = nf;
        if ((q_out && nq > q_cap) || (f_out && nf > f_cap)) throw OFail{TDLB_EINVAL, "output capacity too small"};
    });
}

}  // extern "C"
