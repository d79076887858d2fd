// The zone of a split step: the flag words (32 cells of a row, Dims::word) that
// hold a cell some forcing pass of the resident markers can touch, at any
// impeller angle, and for Esotwist the periodic neighbours of such cells (an
// Esotwist location of a stencil cell is also a location of its neighbours in
// the other parity). Built on the device: the host pass over the lattice's bits
// that this replaces took half a second for a 400^3 tank, these launches read
// the flags once (8 MB).
#include "tdlb_kernels.cuh"

namespace tdlb {

__global__ void __launch_bounds__(256) k_zone_core(Dims g, const uint32_t* __restrict__ mask_static,
                                                   const double2* __restrict__ ring, double ci, double ck,
                                                   uint32_t* __restrict__ core) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= g.rows() * g.jw) return;
    uint32_t bits = mask_static[t];
    const long long row = t / g.jw;
    const int j0 = (int)(t - row * g.jw) * 32;
    const int i = (int)(row / g.nz), k = (int)(row - (long long)i * g.nz);
    const double d = sqrt((i - ci) * (i - ci) + (k - ck) * (k - ck));
    if (ring)
        for (int b = 0; b < 32 && j0 + b < g.ny; b++) {
            const double2 r = ring[j0 + b];
            if (r.y >= 0.0 && d >= r.x && d <= r.y) bits |= 1u << b;
        }
    core[t] = bits;
}

__global__ void __launch_bounds__(256) k_zone_words(Dims g, const uint32_t* __restrict__ core, int neighbours,
                                                    uint8_t* __restrict__ skip) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= g.rows() * g.jw) return;
    if (!neighbours) {
        skip[t] = core[t] != 0u;
        return;
    }
    const long long row = t / g.jw;
    const int w = (int)(t - row * g.jw);
    const int i = (int)(row / g.nz), k = (int)(row - (long long)i * g.nz);
    const int last = (g.ny - 1) >> 5;                     // the word of j = ny - 1
    const int below = w == 0 ? last : w - 1, below_bit = w == 0 ? (g.ny - 1) & 31 : 31;
    const int above = w == last ? 0 : w + 1;
    uint32_t any = 0;
    for (int di = -1; di <= 1; di++)
        for (int dk = -1; dk <= 1; dk++) {
            const int a = (i + di + g.nx) % g.nx, c = (k + dk + g.nz) % g.nz;
            const uint32_t* r = core + ((long long)a * g.nz + c) * g.jw;
            any |= r[w] | ((r[below] >> below_bit) & 1u) | (r[above] & 1u);
        }
    skip[t] = any != 0u;
}

__global__ void __launch_bounds__(256) k_zone_box(Dims g, const int* __restrict__ cells, int n,
                                                  uint32_t* __restrict__ except, uint8_t* __restrict__ skip) {
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (t >= n) return;
    const int e = cells[t], row = e / g.jp, j = e - row * g.jp;
    const long long w = (long long)row * g.jw + (j >> 5);
    if (except) atomicOr(except + w, 1u << (j & 31));
    if (skip) skip[w] = 1;
}

static unsigned words_grid(const Dims& g) { return (unsigned)((g.rows() * g.jw + 255) / 256); }

cudaError_t launch_zone_core(const Dims& g, const uint32_t* mask_static, const double2* ring, double ci, double ck,
                             uint32_t* core, cudaStream_t st) {
    k_zone_core<<<words_grid(g), 256, 0, st>>>(g, mask_static, ring, ci, ck, core);
    return cudaGetLastError();
}
cudaError_t launch_zone_words(const Dims& g, const uint32_t* core, int neighbours, uint8_t* skip, cudaStream_t st) {
    k_zone_words<<<words_grid(g), 256, 0, st>>>(g, core, neighbours, skip);
    return cudaGetLastError();
}
cudaError_t launch_zone_box(const Dims& g, const int* cells, int n, uint32_t* except, uint8_t* skip, cudaStream_t st) {
    if (n > 0) k_zone_box<<<(n + 255) / 256, 256, 0, st>>>(g, cells, n, except, skip);
    return cudaGetLastError();
}

}  // namespace tdlb
